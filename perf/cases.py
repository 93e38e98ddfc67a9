"""What a program has this framework do, as cases that can be timed and checked.

Six kinds of call, each through a public entry point:

``linear``  one NVFP4 W4A4 linear of a model, bf16 tokens in, through the dispatch that a model runner
            calls (``nvfp4r.ops.linear_auto``): single-token decode, batched decode, prompts.
``gemm``    the two raw operators of a program that keeps its activations quantized:
            ``nvfp4r.quant`` (swizzled scales) and ``nvfp4r.gemm``.
``gemv``    the raw operator ``nvfp4r.gemv`` on pre-quantized tokens that share one weight.
``reset``   one step of the ReSET logits processor for a batch of requests in mid-generation.
``sample``  one id per row from the top-k / top-p set of its logits.
``decode``  a whole token of a Qwen3-shaped model from its CUDA graph, to the logits.

Weights are N(0, 0.02) and activations N(0, 1) with 0.1 % of the channels raised twentyfold, both
quantized per 16 elements under a global scale of 6 * 448 / amax; logits are N(0, 3) with one peaked
token per row. The shapes are the linears of Qwen3-8B, 14B and 32B and a vocabulary of 151936.
"""

from __future__ import annotations

import ctypes

import torch

from reset_b200 import _lib, capi
from reset_b200.decode import QWEN3_8B, DecodeConfig, DecodeStep
from reset_b200.nvfp4r import ops

VOCAB = 151936
_OUT = {"bf16": torch.bfloat16, "fp16": torch.float16, "fp32": torch.float32}
_E2M1 = (0.0, 0.5, 1.0, 1.5, 2.0, 3.0, 4.0, 6.0)
_WINDOW, _TAU0, _T_HIGH, _T_LOW = 32, 0.5505, 1.0, 0.1


def listed():
    return [
        # the smallest linear of a decode step, one request: latency and the launch count
        {"name": "o_proj 4096x4096 M1", "kind": "linear", "M": 1, "N": 4096, "K": 4096, "out": "bf16"},
        # the longest rows of a decode step, one request
        {"name": "down 5120x25600 M1", "kind": "linear", "M": 1, "N": 5120, "K": 25600, "out": "bf16"},
        # the widest linear of a decode step, a few requests
        {"name": "gate_up 24576x4096 M8", "kind": "linear", "M": 8, "N": 24576, "K": 4096, "out": "bf16"},
        # batched decode, sixteen requests
        {"name": "gate_up 34816x5120 M16", "kind": "linear", "M": 16, "N": 34816, "K": 5120, "out": "bf16"},
        # batched decode with a ragged number of requests
        {"name": "qkv 10240x5120 M45", "kind": "linear", "M": 45, "N": 10240, "K": 5120, "out": "bf16"},
        # a short prompt of odd length
        {"name": "qkv 6144x4096 M333", "kind": "linear", "M": 333, "N": 6144, "K": 4096, "out": "bf16"},
        # a prompt chunk: the largest call
        {"name": "gate_up 24576x4096 M2048", "kind": "linear", "M": 2048, "N": 24576, "K": 4096, "out": "bf16"},
        # quantized activations kept by the program: quantizer, then the tensor-core operator
        {"name": "quant+gemm 4096x12288 M128", "kind": "gemm", "M": 128, "N": 4096, "K": 12288, "out": "fp16"},
        # the raw GEMV operator on two pre-quantized tokens
        {"name": "gemv 7168x5120 L2", "kind": "gemv", "M": 2, "N": 7168, "K": 5120, "out": "fp16"},
        # the logits processor for a batch of requests
        {"name": "reset step B8", "kind": "reset", "B": 8, "V": VOCAB},
        # the sampler behind it
        {"name": "sample B8 top-k 20 top-p 0.95", "kind": "sample", "B": 8, "V": VOCAB, "top_k": 20, "top_p": 0.95},
        # a whole token of a model of the 8B geometry, four layers deep, context 2048
        {"name": "decode step 4 layers", "kind": "decode", "layers": 4, "context": 2048},
    ]


def _log_int(rng, lo, hi, step=1):
    v = lo * (hi / lo) ** rng.random()
    return max(lo, min(hi, int(v / step + 0.5) * step))


def draw(rng):
    kind = rng.choice(["linear"] * 5 + ["gemm", "gemm", "gemv", "reset", "sample"])
    if kind == "reset":
        return {"kind": kind, "B": _log_int(rng, 1, 32), "V": rng.choice([VOCAB, VOCAB, _log_int(rng, 32000, VOCAB)])}
    if kind == "sample":
        top_k, top_p = rng.choice([(20, 0.95), (0, 0.9), (50, 1.0), (rng.randint(1, 200), 0.5 + 0.49 * rng.random())])
        return {"kind": kind, "B": _log_int(rng, 1, 32), "V": rng.choice([VOCAB, _log_int(rng, 32000, VOCAB)]),
                "top_k": top_k, "top_p": round(top_p, 3)}
    if kind == "gemv":
        return {"kind": kind, "M": rng.randint(1, 8), "N": _log_int(rng, 640, 25600, rng.choice([4, 128])),
                "K": _log_int(rng, 1024, 12288, 32), "out": rng.choice(["fp16", "bf16"])}
    if kind == "gemm":
        return {"kind": kind, "M": _log_int(rng, 1, 1024), "N": _log_int(rng, 640, 16384, 128),
                "K": _log_int(rng, 1024, 12288, 256), "out": rng.choice(["fp16", "bf16"])}
    M = _log_int(rng, 1, 2048)
    if M <= 16 and rng.random() < 0.15:                      # a layer whose sizes no tile divides
        return {"kind": kind, "M": M, "N": _log_int(rng, 500, 8192), "K": _log_int(rng, 1024, 8192, 32), "out": "bf16"}
    return {"kind": kind, "M": M, "N": _log_int(rng, 1024, 24576, 128), "K": _log_int(rng, 1024, 4096, 128) if M > 64
            else _log_int(rng, 1024, 7168, 128), "out": rng.choice(["bf16", "bf16", "bf16", "fp16", "fp32"])}


# ---- inputs ---------------------------------------------------------------------------------------


def _weight_bf16(case, gen):
    return (torch.randn(case["N"], case["K"], device="cuda", generator=gen) * 0.02).to(torch.bfloat16)


def _tokens_bf16(case, gen):
    x = torch.randn(case["M"], case["K"], device="cuda", generator=gen)
    n = max(1, round(case["K"] * 0.001))
    x[:, torch.randperm(case["K"], device="cuda", generator=gen)[:n]] *= 20.0
    return x.to(torch.bfloat16)


def _quantize(x, gs_inv):
    """[R, K] bf16 -> e2m1 codes one per byte [R, K] and e4m3 scales [R, K/16], IEEE fp32 throughout:
    scale = e4m3(gs_inv * (amax / 6)), code = e2m1(x / (scale / gs_inv)), ties to even."""
    R, K = x.shape
    codes = torch.empty(R, K, dtype=torch.uint8, device=x.device)
    scales = torch.empty(R, K // 16, dtype=torch.float8_e4m3fn, device=x.device)
    rcp = torch.ones((), device=x.device) / gs_inv
    for i in range(0, R, 4096):
        b = x[i:i + 4096].float().view(-1, K // 16, 16)
        s = (gs_inv * (b.abs().amax(-1) * torch.tensor(1.0 / 6.0, device=x.device))).clamp(max=448.0)
        s = s.to(torch.float8_e4m3fn)
        scales[i:i + 4096] = s
        d = s.float() * rcp
        r = torch.where(d == 0, torch.zeros_like(d), 1.0 / d)
        y = b * r[..., None]
        a = y.abs()
        c = ((a > 0.25).to(torch.uint8) + (a >= 0.75).to(torch.uint8) + (a > 1.25).to(torch.uint8)
             + (a >= 1.75).to(torch.uint8) + (a > 2.5).to(torch.uint8) + (a >= 3.5).to(torch.uint8)
             + (a > 5.0).to(torch.uint8))
        codes[i:i + 4096] = (c | (torch.signbit(y).to(torch.uint8) << 3)).view(-1, K)
    return codes, scales


def _gs_inv(t):
    return (6.0 * 448.0 / t.float().abs().amax()).reshape(1)


def _linear_inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    w = _weight_bf16(case, gen)
    w_inv = _gs_inv(w)
    codes, scales = _quantize(w, w_inv)
    x = _tokens_bf16(case, gen)
    x_inv = _gs_inv(x)
    return codes, scales, x, x_inv, float(1.0 / (w_inv.double() * x_inv.double()))


def _packed_codes(codes):
    return (codes[:, 0::2] | (codes[:, 1::2] << 4)).contiguous()


def _prepare_linear(case, seed):
    codes, scales, x, x_inv, alpha = _linear_inputs(case, seed)
    st = {"w": _packed_codes(codes), "s": scales.view(torch.uint8), "x": x, "gs": x_inv, "alpha": alpha,
          "out": _OUT[case["out"]], "N": case["N"], "packed": None}
    if case["kind"] == "linear" and case["N"] % 128 == 0 and case["K"] % 128 == 0:
        st["packed"] = ops.pack_weight(st["w"], st["s"])
    if case["kind"] == "gemm":
        st["s"] = capi.swizzle_blockscale(st["s"])
        st["C"] = torch.empty(case["M"], case["N"], dtype=st["out"], device="cuda")
    if case["kind"] == "gemv":
        q, qs = _quantize(x, x_inv)
        M = case["M"]
        st["x"] = _packed_codes(q)[:, None]
        st["xs"] = qs.view(torch.uint8)[:, None].contiguous()
        st["w"] = st["w"][None].expand(M, -1, -1)
        st["s"] = st["s"][None].expand(M, -1, -1)
        st["C"] = torch.empty(M, case["N"], dtype=st["out"], device="cuda")
    return st


def _logits(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    B, V = case["B"], case["V"]
    x = torch.randn(B, V, device="cuda", generator=gen) * 3.0
    peak = torch.randint(0, V, (B, 1), device="cuda", generator=gen)
    # half of the rows are unsure of the token (entropy of several nats), half are confident
    sure = torch.rand(B, 1, device="cuda", generator=gen) < 0.5
    return x.scatter_(1, peak, torch.where(sure, 30.0, 12.0).expand(B, 1).contiguous())


def _history(case, seed):
    """Requests in mid-generation: the last 32 entropies, the open step's and the running sums."""
    rows = []
    g = torch.Generator().manual_seed(seed + 1)
    for _ in range(case["B"]):
        recent = (0.05 + 0.9 * torch.rand(_WINDOW, generator=g)).tolist()
        total = 40 + int(torch.randint(0, 400, (1,), generator=g))
        steps = int(torch.randint(0, 40, (1,), generator=g))
        rows.append({"recent": recent, "head": int(torch.randint(0, 64, (1,), generator=g)), "total": total,
                     "total_sum": total * (0.3 + 0.4 * float(torch.rand(1, generator=g))), "steps": steps,
                     "step_sum": steps * (0.3 + 0.4 * float(torch.rand(1, generator=g)))})
    return rows


def _state_record(h):
    st = _lib.ResetState()
    for i, e in enumerate(h["recent"]):
        st.window_buf[(h["head"] + i) % 64] = e
    st.step_sum, st.total_sum, st.total_count = h["step_sum"], h["total_sum"], h["total"]
    st.step_count, st.window_count, st.window_head = h["steps"], _WINDOW, h["head"]
    return st


def _bytes(records):
    return torch.frombuffer(bytearray(b"".join(bytes(r) for r in records)), dtype=torch.uint8).cuda()


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("linear", "gemm", "gemv"):
        return dict(_prepare_linear(case, seed), kind=kind)
    if kind == "reset":
        B = case["B"]
        params = [_lib.ResetParams(_T_HIGH, _T_LOW, _TAU0, _WINDOW, 0)] * B
        return {"kind": kind, "logits": _logits(case, seed), "states": _bytes(map(_state_record, _history(case, seed))),
                "params": _bytes(params), "ws": capi.reset_workspace(B, "cuda"),
                "decisions": torch.zeros(B * ctypes.sizeof(_lib.ResetDecision), dtype=torch.uint8, device="cuda")}
    if kind == "sample":
        return {"kind": kind, "logits": _logits(case, seed), "top_k": case["top_k"], "top_p": case["top_p"],
                "seed": seed, "ws": capi.sample_workspace(case["B"], "cuda")}
    cfg = DecodeConfig("Qwen3-8B geometry", case["layers"], QWEN3_8B.hidden, QWEN3_8B.q_heads, QWEN3_8B.kv_heads,
                       QWEN3_8B.head_dim, QWEN3_8B.intermediate, QWEN3_8B.vocab, context=case["context"])
    step = DecodeStep(cfg, "cuda", seed=seed)
    step.capture()
    return {"kind": kind, "step": step}


# ---- one pass -------------------------------------------------------------------------------------


def run(st):
    kind = st["kind"]
    if kind == "linear":
        return ops.linear_auto(st["x"], st["gs"], st["w"], st["s"], st["packed"], st["N"], st["alpha"], st["out"])
    if kind == "gemm":
        codes, scales = ops.quant(st["x"], st["gs"], swizzled=True)
        return codes, scales, ops.gemm(codes, st["w"], scales, st["s"], st["C"], st["alpha"])
    if kind == "gemv":
        return ops.gemv(st["w"], st["s"], st["x"], st["xs"], out=st["C"], alpha=st["alpha"])
    if kind == "reset":
        # an engine writes fresh logits every step; the copies stand for that, and keep a pass repeatable
        logits, states = st["logits"].clone(), st["states"].clone()
        capi.reset_step_per_request(logits, states, st["params"], decisions=st["decisions"], workspace=st["ws"])
        B = logits.shape[0]
        return (logits, st["decisions"].view(torch.float64).view(B, -1)[:, :4],
                states.view(torch.float64).view(B, -1)[:, :66], states.view(torch.int32).view(B, -1)[:, 132:])
    if kind == "sample":
        draws = torch.zeros(st["logits"].shape[0], dtype=torch.int64, device="cuda")     # the first draw of a request
        ids = capi.sample(st["logits"], draws, seed=st["seed"], top_k=st["top_k"], top_p=st["top_p"], workspace=st["ws"])
        return ids, draws
    step = st["step"]
    step.replay()
    return step.logits_local, [(layer["k"], layer["v"]) for layer in step.layers]


# ---- what a pass cannot do without, and what it returns ---------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "reset":       # each logit read and written once, about ten operations for its share of the entropy
        return {"bytes": case["B"] * case["V"] * 8, "flops": 10 * case["B"] * case["V"]}
    if kind == "sample":
        return {"bytes": case["B"] * case["V"] * 4, "flops": 5 * case["B"] * case["V"]}
    if kind == "decode":
        c = QWEN3_8B
        qkv, q = (c.q_heads + 2 * c.kv_heads) * c.head_dim, c.q_heads * c.head_dim
        elems = case["layers"] * (qkv * c.hidden + q * c.hidden + 3 * c.hidden * c.intermediate)
        kv = case["layers"] * 2 * c.kv_heads * case["context"] * c.head_dim
        return {"bytes": elems * 9 // 16 + 2 * kv + 2 * c.vocab * c.hidden + 4 * c.vocab,
                "flops": 2 * (elems + c.vocab * c.hidden) + 4 * case["layers"] * c.q_heads * case["context"] * c.head_dim}
    M, N, K = case["M"], case["N"], case["K"]
    size = 4 if case["out"] == "fp32" else 2
    tokens = M * K * 9 // 16 if kind == "gemv" else 2 * M * K
    if kind == "gemm":
        tokens += M * K * 9 // 16                            # the codes and scales are outputs too
    return {"bytes": N * K * 9 // 16 + tokens + M * N * size, "flops": 2 * M * N * K}


def tolerance(case):
    kind = case["kind"]
    if kind == "sample":
        return "exact"
    if kind == "reset":
        return {"rel": 1e-5, "max": 1e-4}
    if kind == "decode":
        return {"rel": 0.03, "max": 0.5}
    # a bf16 / fp16 result is half a unit off the exact sum; codes and scale bytes are exact
    return {"bf16": {"rel": 7e-3, "max": 1.6e-2}, "fp16": {"rel": 1e-3, "max": 2e-3},
            "fp32": {"rel": 1e-5, "max": 1e-4}}[case["out"]]


def _dequant(codes, scales):
    table = torch.tensor(_E2M1 + tuple(-v for v in _E2M1), dtype=torch.float64, device=codes.device)
    v = table[codes.long()].view(codes.shape[0], -1, 16) * scales.double()[..., None]
    return v.view(codes.shape)


def _exact_linear(case, seed):
    codes, scales, x, x_inv, alpha = _linear_inputs(case, seed)
    q = _dequant(*_quantize(x, x_inv))
    out = torch.empty(case["M"], case["N"], dtype=torch.float64, device="cuda")
    for i in range(0, case["N"], 2048):
        out[:, i:i + 2048] = q @ _dequant(codes[i:i + 2048], scales[i:i + 2048]).t()
    return out * alpha


def exact(case, seed):
    kind = case["kind"]
    if kind in ("linear", "gemv"):
        return _exact_linear(case, seed)
    if kind == "gemm":
        return None, None, _exact_linear(case, seed)
    if kind == "reset":
        x = _logits(case, seed).double()
        p = torch.softmax(x, dim=-1)
        ent = (-(p * p.clamp(min=1e-10).log()).sum(-1)).cpu().tolist()
        temps, decisions, sums = [], [], []
        for e, h in zip(ent, _history(case, seed)):
            h_step = sum(h["recent"]) / _WINDOW if h["steps"] < _WINDOW else h["step_sum"] / h["steps"]
            h_bar = h["total_sum"] / h["total"]
            temps.append(_T_HIGH if e >= (h_step if h_step > h_bar else _TAU0) else _T_LOW)
            decisions.append([e, h_step, h_bar, temps[-1]])
            st = _state_record(h)
            st.window_buf[(h["head"] + _WINDOW) % 64] = e        # the oldest leaves, the new one is appended
            sums.append(list(st.window_buf) + [h["step_sum"] + e, h["total_sum"] + e])
        f64 = dict(dtype=torch.float64, device="cuda")
        return x / torch.tensor(temps, **f64)[:, None], torch.tensor(decisions, **f64), torch.tensor(sums, **f64), None
    return None     # sampled ids have no such value, and a chain of quantized layers has none beyond its roundings
