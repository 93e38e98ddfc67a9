"""GPU parity of the many-token tensor-core kernel (``gemm_large.cu``) against the CPU oracle: tile edges
and remainders in tokens and K, both schedules (whole tiles, stream-K), both operand forms (packed
weight through ``torch.ops.nvfp4r.linear_packed``, row-major operands through ``nvfp4r_gemm``), every
output type and layout. Products of e2m1 codes and e4m3 scales are exact and sums are fp32: rel-L2 <=
1e-5 against the float64 dequantise-matmul, the bound of the other tensor-core kernels; 16-bit outputs
add half a unit in the last place per element (2^-8 of it for the 8 significant bits of bf16, 2^-11 for
the 11 of fp16)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from oracle import nvfp4 as onv
from helpers import cuda, make_activation, rel_l2

pytestmark = pytest.mark.gpu

F32 = 2


@pytest.fixture(scope="module")
def capi():
    import reset_b200.nvfp4r  # noqa: F401  (registers the operators)
    from reset_b200 import capi as c
    return c


@pytest.fixture(autouse=True)
def _tuning():
    from reset_b200 import _lib
    yield
    _lib.lib().nvfp4r_set_gemm_large_tuning(0, 0, -1)


def _tune(min_m, bn, sk):
    from reset_b200 import _lib
    _lib.check(_lib.lib().nvfp4r_set_gemm_large_tuning(min_m, bn, sk), "tuning")


def _case(M, N, K, seed):
    w, ws = onv.random_nvfp4((N,), K, seed=seed)
    xb = make_activation(M, K, seed=seed + 1)
    xc, xsf = onv.quantize_nvfp4(xb.float().numpy(), 48.0)
    return w, ws, xb, torch.tensor([48.0], device="cuda"), onv.linear_f64(w, ws, xc, xsf, alpha=0.5)


def _packed(capi, w, ws, xb, gs, N, dtype=F32):
    packed = capi.pack_weight(cuda(w), cuda(ws))
    return torch.ops.nvfp4r.linear_packed(xb, gs, packed, N, 0.5, dtype, 0)


@pytest.mark.parametrize("bn,sk", [(0, -1), (16, 0), (64, 1), (112, 0), (112, 1), (128, 0), (128, 1), (176, 0), (256, 0),
                                   (256, 1)])
@pytest.mark.parametrize("M,N,K", [(33, 128, 128), (45, 2560, 5120), (128, 384, 640), (129, 256, 1024), (257, 1920, 5760)])
def test_packed_tiles_and_schedules(capi, M, N, K, bn, sk):
    _tune(1, bn, sk if sk != 1 or (N // 128) * ((K + 255) // 256) >= 296 else -1)
    w, ws, xb, gs, exact = _case(M, N, K, seed=M + K)
    x = torch.empty(M, K + 24, dtype=torch.bfloat16, device="cuda")[:, :K]     # rows further apart than K
    x.copy_(xb)
    a = _packed(capi, w, ws, x, gs, N)
    b = _packed(capi, w, ws, x, gs, N)
    assert torch.equal(a, b)                                                   # does not depend on arrival order
    assert rel_l2(a.cpu().numpy(), exact) <= 1e-5


def _mixed_plan(M, N, K, bn):
    """True when the plan is whole tiles first, stream-K over the tiles that are left: read off the size of the scratch,
    tokens + 4 bytes a shared tile (in 256s) + two partial tiles for each of the CTAs that share."""
    from reset_b200 import _lib
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    blocks, tiles = (K + 255) // 256, -(-M // bn) * (N // 128)
    tokens = -(-(-(-M // bn) * blocks * (bn * 128 + -(-bn // 128) * 2048)) // 256) * 256
    tickets = (_lib.lib().nvfp4r_linear_packed_scratch_bytes(M, N, K) - tokens) % (2 * bn * 512)
    return tiles > sms and 0 < tickets <= -(-(tiles - sms) * 4 // 256) * 256


@pytest.mark.parametrize("M,N,K,bn", [(256, 2560, 512, 16), (130, 5120, 640, 16), (33, 20480, 1024, 16), (257, 20480, 512, 256),
                                      (130, 20480, 1024, 128)])
def test_whole_tiles_then_stream_k(capi, M, N, K, bn):
    """A CTA crosses from whole tiles to a range of the tiles that are left (with the ring and, above 128 tokens a
    tile, the one accumulator carried across); tickets and partial sums are counted from the first shared tile."""
    _tune(1, bn, 1)
    assert _mixed_plan(M, N, K, bn)
    w, ws, xb, gs, exact = _case(M, N, K, seed=M + bn)
    a = _packed(capi, w, ws, xb.cuda(), gs, N)
    assert torch.equal(a, _packed(capi, w, ws, xb.cuda(), gs, N))
    assert rel_l2(a.cpu().numpy(), exact) <= 1e-5
    if bn < 128 or K % 256:
        return
    xc, xsf = capi.quant(xb.cuda(), gs, swizzled=True)
    wksp = torch.zeros(64 << 20, dtype=torch.uint8, device="cuda")
    for _ in range(2):
        C = torch.full((M, N), float("nan"), device="cuda")
        capi.gemm(xc, cuda(w), xsf, cuda(onv.swizzle_blockscale(ws)), C, 0.5, wksp, n_major=False)
        assert rel_l2(C.cpu().numpy(), exact) <= 1e-5
    assert not wksp[:16384].any()


@pytest.mark.parametrize("parts", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("M,N,K,bn", [(1, 256, 2048, 16), (45, 384, 1920, 48), (100, 128, 4224, 112), (129, 640, 2304, 80),
                                      (200, 256, 2176, 208), (300, 2560, 2048, 128)])
def test_cluster_split(capi, M, N, K, bn, parts):
    """One tile per cluster: more parts than 16-token columns to sum (parts without any), a ragged last part, shares of
    K that differ by a block, a last block of half the steps, more clusters than fit at once."""
    _tune(1, bn, parts)
    w, ws, xb, gs, exact = _case(M, N, K, seed=M + parts)
    a = _packed(capi, w, ws, xb.cuda(), gs, N)
    assert torch.equal(a, _packed(capi, w, ws, xb.cuda(), gs, N))
    assert rel_l2(a.cpu().numpy(), exact) <= 1e-5
    assert rel_l2(_packed(capi, w, ws, xb.cuda(), gs, N, 0).double().cpu().numpy(), exact) <= 2.0 ** -8
    if K % 256 or (M > bn and bn % 128):
        return
    xc, xsf = capi.quant(xb.cuda(), gs, swizzled=True)
    wksp = torch.zeros(1 << 20, dtype=torch.int64, device="cuda")
    for n_major in (True, False):
        C = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
        capi.gemm(xc, cuda(w), xsf, cuda(onv.swizzle_blockscale(ws)), C, 0.5, wksp, n_major=n_major)
        got = C.double().cpu().numpy()
        assert rel_l2(got.reshape(N, M).T if n_major else got, exact) <= 2.0 ** -11
    assert not wksp.any()                                                  # no partial sums in memory


@pytest.mark.parametrize("M,N,K,bn", [(1, 128, 256, 16), (45, 384, 640, 48), (200, 256, 4224, 208), (300, 2560, 2048, 256),
                                      (257, 20480, 512, 128), (600, 10368, 896, 192),
                                      (700, 10368, 1280, 240), (1000, 10240, 768, 256), (1000, 10240, 768, 224)])
def test_pairs_of_sms(capi, M, N, K, bn):
    """Two CTAs on one tile of 256 weight rows: an odd number of row tiles (the last pair has one), more pairs than fit at
    once with accumulators side by side and overlapping (by 16 and 48 tokens), a last block of half the steps, fewer blocks than stages."""
    _tune(1, bn, 9)
    w, ws, xb, gs, exact = _case(M, N, K, seed=M + bn)
    a = _packed(capi, w, ws, xb.cuda(), gs, N)
    assert torch.equal(a, _packed(capi, w, ws, xb.cuda(), gs, N))
    assert rel_l2(a.cpu().numpy(), exact) <= 1e-5
    assert rel_l2(_packed(capi, w, ws, xb.cuda(), gs, N, 0).double().cpu().numpy(), exact) <= 2.0 ** -8
    if K % 256 or (M > bn and bn % 128):
        return
    xc, xsf = capi.quant(xb.cuda(), gs, swizzled=True)
    wksp = torch.zeros(1 << 20, dtype=torch.int64, device="cuda")
    for n_major in (True, False):
        C = torch.full((M, N), float("nan"), dtype=torch.float16, device="cuda")
        capi.gemm(xc, cuda(w), xsf, cuda(onv.swizzle_blockscale(ws)), C, 0.5, wksp, n_major=n_major)
        got = C.double().cpu().numpy()
        assert rel_l2(got.reshape(N, M).T if n_major else got, exact) <= 2.0 ** -11


@pytest.mark.parametrize("N,K,first", [(1536, 256, 13), (4096, 256, 17), (384, 256, 17), (256, 256, 25), (256, 384, 33)])
def test_first_token_count_follows_the_shape(capi, N, K, first):
    """Both sides of the line between the decode kernel and this one, per shape class, give the same product."""
    from reset_b200 import _lib
    for M in (first - 1, first):
        assert (_lib.lib().nvfp4r_linear_packed_scratch_bytes(M, N, K) > 0) == (M >= first)
        w, ws, xb, gs, exact = _case(M, N, K, seed=M)
        assert rel_l2(_packed(capi, w, ws, xb.cuda(), gs, N).cpu().numpy(), exact) <= 1e-5


@pytest.mark.parametrize("M", [1, 2, 15, 16, 17, 31, 32, 47, 64, 65, 96, 127, 200, 255, 256, 300, 511, 513, 777])
def test_packed_token_counts_stay_inside_the_output(capi, M):
    from reset_b200 import _lib
    _tune(1, 0, -1)
    N, K = 256, 768
    w, ws, xb, gs, exact = _case(M, N, K, seed=M)
    packed, x = capi.pack_weight(cuda(w), cuda(ws)), xb.cuda()
    lib = _lib.lib()
    n = lib.nvfp4r_linear_packed_scratch_bytes(M, N, K)
    scratch = torch.full((n + 512,), 0x7F, dtype=torch.uint8, device="cuda")   # NaN scales wherever nothing is written
    out = torch.full((M * N + 512,), 7.0, device="cuda")
    st = lib.nvfp4r_linear_packed_scratch(x.data_ptr(), K, M, K, gs.data_ptr(), packed.data_ptr(), N, 0.5,
                                          out.data_ptr() + 1024, F32, 0, scratch.data_ptr() + 256, n,
                                          torch.cuda.current_stream().cuda_stream)
    _lib.check(st, "linear_packed_scratch")
    got = out.cpu().numpy()
    assert (got[:256] == 7.0).all() and (got[256 + M * N:] == 7.0).all()
    s = scratch.cpu().numpy()
    assert (s[:256] == 0x7F).all() and (s[256 + n:] == 0x7F).all()
    assert rel_l2(got[256:256 + M * N].reshape(M, N), exact) <= 1e-5


@pytest.mark.parametrize("M,N,K", [(40, 640, 8192), (13, 19456, 2048)])
def test_scratch_entry_takes_shapes_where_the_other_is_faster(capi, M, N, K):
    """The route is advice: a program that calls with the scratch all the same is served."""
    from reset_b200 import _lib
    lib = _lib.lib()
    n = lib.nvfp4r_linear_packed_scratch_bytes(M, N, K)
    assert n > 0 and lib.nvfp4r_linear_packed_route(M, N, K) == 0
    w, ws, xb, gs, exact = _case(M, N, K, seed=M)
    packed, x = capi.pack_weight(cuda(w), cuda(ws)), xb.cuda()
    scratch, out = torch.empty(n, dtype=torch.uint8, device="cuda"), torch.full((M, N), float("nan"), device="cuda")
    args = [x.data_ptr(), K, M, K, gs.data_ptr(), packed.data_ptr(), N, 0.5, out.data_ptr(), F32, 0, scratch.data_ptr(), n,
            torch.cuda.current_stream().cuda_stream]
    _lib.check(lib.nvfp4r_linear_packed_scratch(*args), "linear_packed_scratch")
    assert rel_l2(out.cpu().numpy(), exact) <= 1e-5
    args[2] = 12                                             # fewer tokens than any class starts with
    assert lib.nvfp4r_linear_packed_scratch(*args) == -2


_NO_FIXED_BUFFER = """
import sys, torch
import reset_b200.nvfp4r
for M, N, K in ((16, 20480, 2048), (16, 6144, 1024), (33, 1024, 8192)):
    w = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, device="cuda")
    s = torch.full((N, K // 16), 0x38, dtype=torch.uint8, device="cuda")                     # 0x38: scale 1
    packed = torch.ops.nvfp4r.pack_weight(w, s)
    x, gs = torch.full((M, K), 6.0, dtype=torch.bfloat16, device="cuda"), torch.ones(1, device="cuda")   # code 6, scale 1
    call = lambda: torch.ops.nvfp4r.linear_packed(x, gs, packed, N, 1.0, 2, 0)
    if sys.argv[1] == "captured":
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            out = call()
        g.replay()
    else:
        out = call()
    table = torch.tensor([0, .5, 1, 1.5, 2, 3, 4, 6, 0, -.5, -1, -1.5, -2, -3, -4, -6], device="cuda")
    want = 6 * (table[(w & 15).long()].sum(1) + table[(w >> 4).long()].sum(1))
    assert torch.equal(out, want.expand(M, N)), (M, N, K)                                    # sums of halves: exact
"""


@pytest.mark.parametrize("how,megabytes", [("captured", "128"), ("eager", "1")])
def test_many_tokens_need_no_fixed_buffer(how, megabytes):
    """In a process of its own: a captured call that no other came before, and calls for which the fixed buffer (1 MB)
    is too small for the decode kernel's workspace, take this kernel wherever it takes the shape."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", _NO_FIXED_BUFFER, how], env=dict(os.environ, NVFP4R_WORKSPACE_MB=megabytes),
                       cwd=root, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]


@pytest.mark.parametrize("dtype,half_ulp", [(0, 2.0 ** -8), (1, 2.0 ** -11)])
def test_packed_16_bit_outputs_round_once(capi, dtype, half_ulp):
    M, N, K = 131, 384, 1024
    w, ws, xb, gs, exact = _case(M, N, K, seed=5)
    got = _packed(capi, w, ws, xb.cuda(), gs, N, dtype).double().cpu().numpy()
    scale = np.abs(exact) + np.sqrt(np.mean(exact ** 2)) * 1e-3
    assert np.max(np.abs(got - exact) / scale) <= half_ulp * 1.01


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32])
@pytest.mark.parametrize("n_major", [True, False])
@pytest.mark.parametrize("M,N,K,bn,sk", [(33, 128, 256, 0, -1), (40, 2560, 4096, 0, 1), (64, 1280, 8192, 64, 1),
                                         (130, 384, 1024, 128, 0), (300, 1280, 4096, 256, 1), (257, 256, 512, 256, 0)])
def test_gemm_row_major(capi, M, N, K, bn, sk, n_major, dtype):
    _tune(0, bn, sk)
    w, ws, xb, gs, exact = _case(M, N, K, seed=M + N)
    xc, xsf = capi.quant(xb.cuda(), gs, swizzled=True)
    C = torch.full((M, N), float("nan"), dtype=dtype, device="cuda")
    wksp = torch.zeros(16 << 20, dtype=torch.int64, device="cuda")
    capi.gemm(xc, cuda(w), xsf, cuda(onv.swizzle_blockscale(ws)), C, 0.5, wksp, n_major=n_major)
    got = C.double().cpu().numpy()
    got = got.reshape(N, M).T if n_major else got
    assert rel_l2(got, exact) <= {torch.float32: 1e-5, torch.float16: 2.0 ** -11, torch.bfloat16: 2.0 ** -8}[dtype]


@pytest.mark.parametrize("M,bn", [(130, 64), (130, 16), (257, 112), (257, 176), (520, 64)])
def test_gemm_row_major_tiles_start_at_a_scale_chunk(capi, M, bn):
    """Row-major token scales are addressed in chunks of 128 rows: with more than one tile a width asked for by
    tuning is rounded up to that, for a tile may neither read another tile's scales nor past the last chunk."""
    _tune(0, bn, 0)
    N, K = 256, 512
    w, ws, xb, gs, exact = _case(M, N, K, seed=M + bn)
    xc, xsf = capi.quant(xb.cuda(), gs, swizzled=True)
    C = torch.full((M, N), float("nan"), device="cuda")
    wksp = torch.zeros(16 << 20, dtype=torch.uint8, device="cuda")
    capi.gemm(xc, cuda(w), xsf, cuda(onv.swizzle_blockscale(ws)), C, 0.5, wksp, n_major=False)
    assert rel_l2(C.cpu().numpy(), exact) <= 1e-5


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
@pytest.mark.parametrize("M,N,K", [(1, 128, 256), (2, 640, 1024), (7, 384, 4096), (15, 256, 512), (16, 256, 2816), (17, 1280, 768),
                                   (31, 256, 2048), (46, 256, 512), (77, 128, 768), (101, 19072, 256), (333, 640, 512)])
def test_gemm_few_tokens_and_ragged_rows(capi, M, N, K, dtype):
    """Up to 32 tokens, and N-major rows of every alignment (M odd, M % 8 in 2 .. 6): nothing outside the output is
    written, 16-bit results are within half a unit of the exact sum."""
    w, ws, xb, gs, exact = _case(M, N, K, seed=M + N)
    xc, xsf = capi.quant(xb.cuda(), gs, swizzled=True)
    buf = torch.full((M * N + 64,), 7.0, dtype=dtype, device="cuda")
    C, wksp = buf[32:32 + M * N].view(M, N), torch.zeros(16 << 20, dtype=torch.int64, device="cuda")
    for n_major in (True, False):
        capi.gemm(xc, cuda(w), xsf, cuda(onv.swizzle_blockscale(ws)), C, 0.5, wksp, n_major=n_major)
        got = C.double().cpu().numpy()
        got = got.reshape(N, M).T if n_major else got
        scale = np.abs(exact) + np.sqrt(np.mean(exact ** 2)) * 1e-3
        assert np.max(np.abs(got - exact) / scale) <= (2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11) * 1.01
        assert (buf[:32] == 7.0).all() and (buf[32 + M * N:] == 7.0).all()


def test_gemm_output_of_any_alignment(capi):
    """A 2-byte aligned output takes the narrow stores."""
    M, N, K = 48, 256, 512
    w, ws, xb, gs, exact = _case(M, N, K, seed=9)
    xc, xsf = capi.quant(xb.cuda(), gs, swizzled=True)
    buf = torch.zeros(M * N + 1, dtype=torch.float16, device="cuda")
    wksp = torch.zeros(16 << 20, dtype=torch.int64, device="cuda")
    for n_major in (True, False):
        C = buf[1:].view(M, N)
        capi.gemm(xc, cuda(w), xsf, cuda(onv.swizzle_blockscale(ws)), C, 0.5, wksp, n_major=n_major)
        got = C.double().cpu().numpy()
        assert rel_l2(got.reshape(N, M).T if n_major else got, exact) <= 2.0 ** -11


def test_gemm_small_workspace_takes_the_other_kernel(capi):
    """A workspace sized for 32 rows served any M before and still does."""
    M, N, K = 70, 512, 4096
    w, ws, xb, gs, exact = _case(M, N, K, seed=3)
    xc, xsf = capi.quant(xb.cuda(), gs, swizzled=True)
    C = torch.empty((M, N), device="cuda")
    capi.gemm(xc, cuda(w), xsf, cuda(onv.swizzle_blockscale(ws)), C, 0.5, capi.gemm_workspace(32, N, K, "cuda"), n_major=False)
    assert rel_l2(C.cpu().numpy(), exact) <= 1e-5


def test_linear_packed_under_capture(capi):
    M, N, K = 160, 512, 1024
    w, ws, xb, gs, exact = _case(M, N, K, seed=4)
    packed, x = capi.pack_weight(cuda(w), cuda(ws)), xb.cuda()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = torch.ops.nvfp4r.linear_packed(x, gs, packed, N, 0.5, F32, 0)
    for _ in range(3):
        out.zero_()
        g.replay()
        assert rel_l2(out.cpu().numpy(), exact) <= 1e-5


@pytest.mark.parametrize("M,N,K", [(16, 6144, 1024), (32, 1024, 1024), (17, 3072, 1024), (16, 34816, 1024), (32, 8192, 4096)])
def test_eager_and_captured_calls_give_the_same_product(capi, M, N, K):
    """Up to 32 tokens an eager call may take the decode kernel where a captured one takes this one: the operator's
    result is the oracle's either way."""
    from reset_b200 import _lib
    assert _lib.lib().nvfp4r_linear_packed_route(M, N, K) == (2 if K == 4096 else 1 if N < 16 * K else 0)
    w, ws, xb, gs, exact = _case(M, N, K, seed=N % 89)
    packed, x = capi.pack_weight(cuda(w), cuda(ws)), xb.cuda()
    eager = torch.ops.nvfp4r.linear_packed(x, gs, packed, N, 0.5, F32, 0)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        out = torch.ops.nvfp4r.linear_packed(x, gs, packed, N, 0.5, F32, 0)
    g.replay()
    for got in (eager, out):
        assert rel_l2(got.cpu().numpy(), exact) <= 1e-5


@pytest.mark.parametrize("M,dtype", [(1, torch.bfloat16), (32, torch.float16), (32, torch.float32), (33, torch.float16), (300, torch.bfloat16),
                                     (1500, torch.bfloat16)])
def test_gemm_directly_behind_the_quantizer_of_its_weight(capi, M, dtype):
    """The weight is quantized last, into buffers that hold the weight before it, and multiplied at once: the call gives
    what it gives when everything has ended before it."""
    from reset_b200 import _lib
    lib, N, K = _lib.lib(), 2560, 4096
    gen = torch.Generator(device="cuda").manual_seed(M)
    x = torch.randn(M, K, generator=gen, device="cuda").bfloat16()
    weights = [torch.randn(N, K, generator=gen, device="cuda").bfloat16() for _ in range(3)]
    gs = torch.tensor([300.0], device="cuda")
    xc, xsf = capi.quant(x, gs, swizzled=True)
    wc, wsf = torch.empty(N, K // 2, dtype=torch.uint8, device="cuda"), torch.empty(N, K // 16, dtype=torch.uint8, device="cuda")
    wksp = torch.zeros(4 << 20, dtype=torch.int64, device="cuda")

    def quantize(w):
        _lib.check(lib.nvfp4r_quant(w.data_ptr(), K, N, K, gs.data_ptr(), wc.data_ptr(), wsf.data_ptr(), _lib.SF_SWIZZLED, 1,
                                    torch.cuda.current_stream().cuda_stream), "quant")

    def product():
        C = torch.empty((M, N), dtype=dtype, device="cuda")
        capi.gemm(xc, wc, xsf, wsf, C, 1e-5, wksp)
        return C

    want = []
    for w in weights:
        quantize(w)
        torch.cuda.synchronize()
        want.append(product())
        torch.cuda.synchronize()
    assert not torch.equal(want[0], want[1])
    got = []
    for i in range(12):
        quantize(weights[i % 3])
        got.append(product())
    for i in range(12):
        assert torch.equal(got[i], want[i % 3]), i


@pytest.mark.parametrize("bn", [192, 256])                               # accumulators apart, overlapping
@pytest.mark.parametrize("row_major", [False, True])
def test_pairs_hand_stages_and_accumulators_over_in_order(capi, row_major, bn):
    """Many tiles and ring turns a pair, an odd number of row tiles, two weights in turn: every call gives the bits of the first
    one with its weight (the sums have one order), and those of the first are within the bound of the exact product."""
    M, N, K = 1500, 3 * 128 * 31, 2048
    cases = [_case(M, N, K, seed=s) for s in (1, 5)]
    _tune(1, bn, 9)
    x, gs = [c[2].cuda() for c in cases], cases[0][3]
    if row_major:
        operands = [(*capi.quant(x[i], gs, swizzled=True), cuda(cases[i][0]), cuda(onv.swizzle_blockscale(cases[i][1]))) for i in (0, 1)]
        wksp = torch.zeros(1 << 20, dtype=torch.int64, device="cuda")

        def call(i):
            C = torch.empty((M, N), device="cuda")
            xc, xsf, w, ws = operands[i]
            capi.gemm(xc, w, xsf, ws, C, 0.5, wksp, n_major=False)
            return C
    else:
        packed = [capi.pack_weight(cuda(c[0]), cuda(c[1])) for c in cases]

        def call(i):
            return torch.ops.nvfp4r.linear_packed(x[i], gs, packed[i], N, 0.5, F32, 0)
    first = [call(0), call(1)]
    for i in (0, 1):
        assert rel_l2(first[i].cpu().numpy(), cases[i][4]) <= 1e-5
    for r in range(30):
        assert torch.equal(call(r & 1), first[r & 1]), r
