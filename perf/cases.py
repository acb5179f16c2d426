"""Performance cases of the library: the work a host program has it do, through its public calls.

Five kinds of work, each a family of cases with a range of sizes:

  linear   one quantised projection called by itself: activation quantiser + GEMV / GEMM
  decode   a few layers of a decode or verification step, captured once as a CUDA graph and replayed
           per token, the way an engine runs its decode body
  prefill  one dense layer over a prompt chunk, called eagerly
  moe      one mixture-of-experts layer (library layer call) on 1 .. 16,384 tokens
  head     the tied bf16 output head with its arg-max, 1 .. 8 hidden rows

Sizes are those of the repository's benchmark configurations (dense: hidden 3,840, attention 4,096,
QKV 8,192, MLP 15,360; MoE: hidden 2,816, 128 experts top-8 of 704, shared 2,112) plus generic
ones around them, ragged ones included.
"""
import numpy as np
import torch

from gem16_b200 import load
from gem16_b200.moe import MoeLayer, synthetic_weights

F32, BF16 = 0, 1            # GEMB_F32, GEMB_BF16
COMPACT, INTERLEAVED = 0, 1  # scale layouts
EXACT = 0                    # quantiser contract

# Largest magnitudes the static input divisors are set for: normalised activations and GELU products.
ACT_AMAX, PRODUCT_AMAX = 6.0, 16.0
GA, GP = 2688.0 / ACT_AMAX, 2688.0 / PRODUCT_AMAX


def listed():
    return [
        # A single projection of a decode step called by itself from the host (attention output,
        # one token): two short launches, so launch cost and latency count.
        {"name": "linear_fp8_1", "family": "linear", "format": "fp8", "tokens": 1, "rows": 3840, "k": 4096},
        # One NVFP4 linear over a 512-token prompt, the repository's first benchmark configuration.
        {"name": "linear_nvfp4_512", "family": "linear", "format": "nvfp4", "tokens": 512, "rows": 15360, "k": 3840},
        # Batch-1 decode with FP8 weights everywhere: the decode GEMV set (QKV, O, gate/up, down), per-token
        # quantisers included, four layers of it.
        {"name": "decode_fp8_1", "family": "decode", "mlp": "fp8", "tokens": 1, "layers": 4, "hidden": 3840,
         "attention": 4096, "kv": 2048, "inter": 15360},
        # Batch-1 decode of the mixed model: FP8 attention projections, NVFP4 MLP, norms and residuals between.
        {"name": "decode_nvfp4_1", "family": "decode", "mlp": "nvfp4", "tokens": 1, "layers": 4, "hidden": 3840,
         "attention": 4096, "kv": 2048, "inter": 15360},
        # The speculative-decoding verifier: the same layers on five draft tokens at once.
        {"name": "verify_nvfp4_5", "family": "decode", "mlp": "nvfp4", "tokens": 5, "layers": 4, "hidden": 3840,
         "attention": 4096, "kv": 2048, "inter": 15360},
        # Output head of one decode step: one pass over 2 GB of bf16 weights.
        {"name": "head_1", "family": "head", "rows": 1, "vocab": 262144, "hidden": 3840},
        # A short chat prompt through one dense layer: weights dominate, the token count is ragged.
        {"name": "prefill_77", "family": "prefill", "tokens": 77, "hidden": 3840, "attention": 4096, "qkv": 8192, "inter": 15360},
        # A long prompt chunk through one dense layer: the tensor cores' case.
        {"name": "prefill_16384", "family": "prefill", "tokens": 16384, "hidden": 3840, "attention": 4096, "qkv": 8192,
         "inter": 15360},
        # A decode batch of 64 sequences through one MoE layer: about a hundred experts touched.
        {"name": "moe_64", "family": "moe", "tokens": 64, "router": "plain", "hidden": 2816, "experts": 128, "topk": 8,
         "inter": 704, "shared": 2112},
        # A ragged prompt through a layer that routes by the specification's form (normalised and scaled
        # router input, per-expert scales).
        {"name": "moe_spec_3001", "family": "moe", "tokens": 3001, "router": "spec", "hidden": 2816, "experts": 128,
         "topk": 8, "inter": 704, "shared": 2112},
        # A full prefill batch through one MoE layer.
        {"name": "moe_16384", "family": "moe", "tokens": 16384, "router": "plain", "hidden": 2816, "experts": 128,
         "topk": 8, "inter": 704, "shared": 2112},
    ]


def _log_int(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    family = rng.choice(["linear", "decode", "prefill", "moe", "head"])
    if family == "linear":
        fmt = rng.choice(["fp8", "nvfp4"])
        # one token to a prompt chunk; a decode call every third time
        tokens = 1 if rng.random() < 0.33 else _log_int(rng, 9, 4096)
        return {"family": family, "format": fmt, "tokens": tokens, "rows": 8 * _log_int(rng, 128, 1920),
                "k": 64 * _log_int(rng, 16, 160)}
    if family == "decode":
        hidden = 64 * rng.randint(24, 80)
        inter = 64 * rng.randint(2 * hidden // 64, min(4 * hidden // 64, 240))
        mlp = rng.choice(["fp8", "nvfp4", "nvfp4"])
        tokens = rng.choice([1, 1, rng.randint(2, 5)])
        if mlp == "nvfp4" and tokens > 1 and inter <= 8192:
            tokens = rng.randint(2, 8)
        if mlp == "fp8":
            tokens = 1
        return {"family": family, "mlp": mlp, "tokens": tokens, "layers": rng.randint(2, 4), "hidden": hidden,
                "attention": 256 * rng.randint(8, 20), "kv": 256 * rng.randint(2, 8), "inter": inter}
    if family == "prefill":
        hidden = 64 * rng.randint(24, 60)
        return {"family": family, "tokens": _log_int(rng, 17, 12000), "hidden": hidden, "attention": 256 * rng.randint(8, 16),
                "qkv": 256 * rng.randint(12, 32), "inter": 64 * rng.randint(2 * hidden // 64, 4 * hidden // 64)}
    if family == "moe":
        topk = rng.choice([4, 6, 8, 8])
        return {"family": family, "tokens": _log_int(rng, 1, 12000), "router": rng.choice(["plain", "spec"]),
                "hidden": 128 * rng.randint(10, 24), "experts": rng.choice([64, 128, 128]), "topk": topk,
                "inter": 64 * rng.randint(6, 13), "shared": 64 * rng.randint(16, 36)}
    return {"family": family, "rows": rng.randint(1, 8), "vocab": _log_int(rng, 32000, 262000), "hidden": 64 * rng.randint(24, 60)}


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
class _Maker:
    """Seeded tensors and quantised weights on the GPU: activations ~ N(0, 1), weights ~ N(0, 0.02)."""

    def __init__(self, seed):
        self.lib = load()
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.dev)
        self.gen.manual_seed(int(seed))

    def normal(self, *shape, std=1.0):
        return torch.randn(shape, device=self.dev, generator=self.gen) * std

    def bf16(self, *shape, std=1.0):
        return self.normal(*shape, std=std).to(torch.bfloat16).view(torch.int16)

    def norm_weight(self, n):
        return (1.0 + self.normal(n, std=0.1)).to(torch.bfloat16).view(torch.int16)

    def empty(self, *shape, dtype=torch.uint8):
        return torch.empty(shape, dtype=dtype, device=self.dev)

    def zeros(self, n):
        return torch.zeros((n,), dtype=torch.uint8, device=self.dev)

    def scale_bytes(self, rows, k):
        return self.lib.cdll.gemb_interleaved_scale_bytes(rows, k)

    def fp8_weight(self, rows, k):
        w = self.normal(rows, k, std=0.02)
        q, s = self.empty(rows, k), self.empty(rows, dtype=torch.float32)
        self.lib.gemb_fp8_quantize(w, F32, q, s, rows, k, None)
        return q, s.to(torch.bfloat16).view(torch.int16)

    def nvfp4_weight(self, rows, k, layout):
        w = self.normal(rows, k, std=0.02)
        g = float(2688.0 / w.abs().max().item())
        q = self.empty(rows, k // 2)
        s = self.empty(rows, k // 16) if layout == COMPACT else self.zeros(self.scale_bytes(rows, k))
        self.lib.gemb_nvfp4_quantize(w, F32, q, s, rows, k, g, layout, EXACT, None)
        return q, s, g


def _prepare_linear(m, c):
    t, n, k = c["tokens"], c["rows"], c["k"]
    s = {"x": m.bf16(t, k)}
    if c["format"] == "fp8":
        s["w"], s["ws"] = m.fp8_weight(n, k)
        s["xq"], s["xs"] = m.empty(t, k), m.empty(t, dtype=torch.float32)
    else:
        layout = COMPACT if t == 1 else INTERLEAVED
        s["w"], s["ws"], s["gw"] = m.nvfp4_weight(n, k, layout)
        s["xq"] = m.empty(t, k // 2)
        s["xs"] = m.empty(t, k // 16) if t == 1 else m.zeros(m.scale_bytes(t, k))
    s["y"] = m.empty(t, n, dtype=torch.float32 if t == 1 else torch.bfloat16)
    return s


def _run_linear(lib, c, s):
    t, n, k = c["tokens"], c["rows"], c["k"]
    if c["format"] == "fp8":
        lib.gemb_fp8_quantize(s["x"], BF16, s["xq"], s["xs"], t, k, None)
        if t == 1:
            lib.gemb_fp8_gemv(s["xq"], s["xs"], s["w"], s["ws"], s["y"], n, k, None)
        else:
            lib.gemb_fp8_gemm_bf16(s["xq"], s["xs"], s["w"], s["ws"], s["y"], t, n, k, None)
    else:
        lib.gemb_nvfp4_quantize(s["x"], BF16, s["xq"], s["xs"], t, k, GA, COMPACT if t == 1 else INTERLEAVED, EXACT, None)
        if t == 1:
            lib.gemb_nvfp4_gemv(s["xq"], s["xs"], s["w"], s["ws"], s["y"], n, k, GA, s["gw"], None)
        else:
            lib.gemb_nvfp4_gemm_bf16(s["xq"], s["xs"], s["w"], s["ws"], s["y"], t, n, k, GA, s["gw"], None)
    return s["y"]


def _decode_buffers(m, c):
    t, h, a, kv, i = c["tokens"], c["hidden"], c["attention"], c["kv"], c["inter"]
    f32 = torch.float32
    layers = []
    for _ in range(c["layers"]):
        if c["mlp"] == "fp8":
            L = {"qkv": m.fp8_weight(a + 2 * kv, h), "o": m.fp8_weight(h, a), "gate_up": m.fp8_weight(2 * i, h), "down": m.fp8_weight(h, i)}
            L["x"] = {"qkv": m.bf16(1, h), "o": m.bf16(1, a), "gate_up": m.bf16(1, h), "down": m.bf16(1, i)}
            L["xq"] = {n: m.empty(*x.shape) for n, x in L["x"].items()}
            L["xs"] = {n: m.empty(1, dtype=f32) for n in L["x"]}
            L["y"] = {n: m.empty(L[n][0].shape[0], dtype=f32) for n in L["x"]}
        else:
            L = {"q": m.fp8_weight(a, h), "k": m.fp8_weight(kv, h), "v": m.fp8_weight(kv, h), "o": m.fp8_weight(h, a),
                 "gate": m.nvfp4_weight(i, h, COMPACT), "up": m.nvfp4_weight(i, h, COMPACT), "down": m.nvfp4_weight(h, i, COMPACT),
                 "norms": [m.norm_weight(h) for _ in range(4)], "attn": m.normal(t, a),
                 "q_out": m.empty(t, a, dtype=f32), "k_out": m.empty(t, kv, dtype=f32), "v_out": m.empty(t, kv, dtype=f32),
                 "h": m.empty(t, h, dtype=f32)}
        layers.append(L)
    s = {"layers": layers}
    if c["mlp"] == "nvfp4":
        s["x"] = m.bf16(t, h).view(torch.bfloat16).float()
        s["xq"], s["xs"] = m.empty(t, h), m.empty(t, dtype=f32)
        s["aq"], s["as"] = m.empty(t, a), m.empty(t, dtype=f32)
        s["o"], s["mid"], s["d"] = (m.empty(t, h, dtype=f32) for _ in range(3))
        s["hq"], s["hs"] = m.empty(t, h // 2), m.empty(t, h // 16)
        s["p"] = m.empty(t, i, dtype=f32)
        s["pq"], s["ps"] = m.empty(t, i // 2), m.empty(t, i // 16)
    return s


def _decode_calls(lib, c, s, st):
    """The calls of one decode / verification step, in the order the engine's decode body issues them."""
    t, h, a, kv, i = c["tokens"], c["hidden"], c["attention"], c["kv"], c["inter"]
    if c["mlp"] == "fp8":
        for L in s["layers"]:
            for n in ("qkv", "o", "gate_up", "down"):
                w, ws = L[n]
                rows, k = w.shape
                lib.gemb_fp8_quantize(L["x"][n], BF16, L["xq"][n], L["xs"][n], 1, k, st)
                lib.gemb_fp8_gemv(L["xq"][n], L["xs"][n], w, ws, L["y"][n], rows, k, st)
        return
    x, eps = s["x"], 1e-6
    for L in s["layers"]:
        n0, n1, n2, n3 = L["norms"]
        lib.gemb_fp8_rmsnorm_quantize(x, F32, n0, s["xq"], s["xs"], t, h, eps, st)
        q, k, v = L["q"], L["k"], L["v"]
        if t == 1:
            lib.gemb_fp8_gemv_qkv(s["xq"], s["xs"], q[0], q[1], L["q_out"], a, k[0], k[1], L["k_out"], kv, v[0], v[1], L["v_out"], kv,
                                  h, st)
        else:
            lib.gemb_fp8_gemv_qkv_batch(s["xq"], s["xs"], q[0], q[1], L["q_out"], a, k[0], k[1], L["k_out"], kv, v[0], v[1],
                                        L["v_out"], kv, t, h, st)
        # attention itself is not part of the library: its result is a given tensor
        lib.gemb_fp8_quantize(L["attn"], F32, s["aq"], s["as"], t, a, st)
        if t == 1:
            lib.gemb_fp8_gemv(s["aq"], s["as"], L["o"][0], L["o"][1], s["o"], h, a, st)
        else:
            lib.gemb_fp8_gemv_batch(s["aq"], s["as"], L["o"][0], L["o"][1], s["o"], t, h, a, st)
        lib.gemb_rmsnorm_residual(s["o"], F32, n1, x, None, s["mid"], F32, t, h, eps, None, st)
        lib.gemb_nvfp4_rmsnorm_quantize(s["mid"], F32, n2, s["hq"], s["hs"], t, h, eps, GA, COMPACT, EXACT, st)
        (gw, gs, gd), (uw, us, ud), (dw, ds, dd) = L["gate"], L["up"], L["down"]
        if t == 1:
            lib.gemb_nvfp4_gemv_gate_up(s["hq"], s["hs"], gw, gs, uw, us, None, None, s["p"], i, h, GA, gd, GA, ud, st)
        else:
            lib.gemb_nvfp4_gemv_gate_up_batch(s["hq"], s["hs"], gw, gs, uw, us, None, None, s["p"], t, i, h, GA, gd, GA, ud, st)
        lib.gemb_nvfp4_quantize(s["p"], F32, s["pq"], s["ps"], t, i, GP, COMPACT, EXACT, st)
        if t == 1:
            lib.gemb_nvfp4_gemv(s["pq"], s["ps"], dw, ds, s["d"], h, i, GP, dd, st)
        else:
            lib.gemb_nvfp4_gemv_batch(s["pq"], s["ps"], dw, ds, s["d"], t, h, i, GP, dd, st)
        lib.gemb_rmsnorm_residual(s["d"], F32, n3, s["mid"], None, L["h"], F32, t, h, eps, None, st)
        x = L["h"]


def _prepare_decode(m, c):
    s = _decode_buffers(m, c)
    stream = torch.cuda.Stream(device=m.dev)
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        _decode_calls(m.lib, c, s, stream)     # first calls configure the kernels
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        _decode_calls(m.lib, c, s, stream)
    s["graph"] = graph
    return s


def _run_decode(lib, c, s):
    s["graph"].replay()
    if c["mlp"] == "fp8":
        return [[L["y"][n] for n in ("qkv", "o", "gate_up", "down")] for L in s["layers"]]
    return [[L["q_out"], L["k_out"], L["v_out"], L["h"]] for L in s["layers"]]


def _prepare_prefill(m, c):
    t, h, a, qkv, i = c["tokens"], c["hidden"], c["attention"], c["qkv"], c["inter"]
    s = {"x": m.bf16(t, h), "attn": m.bf16(t, a), "norms": [m.norm_weight(h) for _ in range(4)]}
    s["qkv"], s["o"] = m.fp8_weight(qkv, h), m.fp8_weight(h, a)
    (gq, gs, gd), (uq, us, ud) = m.nvfp4_weight(i, h, COMPACT), m.nvfp4_weight(i, h, COMPACT)
    fused, fused_s = m.empty(2 * i, h // 2), m.zeros(m.scale_bytes(2 * i, h))
    m.lib.gemb_nvfp4_pack_gate_up(gq, gs, uq, us, fused, fused_s, i, h, None)
    s["gate_up"], s["down"] = (fused, fused_s, gd, ud), m.nvfp4_weight(h, i, INTERLEAVED)
    bf = torch.bfloat16
    s["xq"], s["xs"] = m.empty(t, h), m.empty(t, dtype=torch.float32)
    s["aq"], s["as"] = m.empty(t, a), m.empty(t, dtype=torch.float32)
    s["y_qkv"], s["y_o"], s["mid"], s["y_d"], s["out"] = m.empty(t, qkv, dtype=bf), *(m.empty(t, h, dtype=bf) for _ in range(4))
    s["hq"], s["hs"] = m.empty(t, h // 2), m.zeros(m.scale_bytes(t, h))
    s["pq"], s["ps"] = m.empty(t, i // 2), m.zeros(m.scale_bytes(t, i))
    return s


def _run_prefill(lib, c, s):
    t, h, a, qkv, i = c["tokens"], c["hidden"], c["attention"], c["qkv"], c["inter"]
    n0, n1, n2, n3 = s["norms"]
    eps = 1e-6
    lib.gemb_fp8_rmsnorm_quantize(s["x"], BF16, n0, s["xq"], s["xs"], t, h, eps, None)
    lib.gemb_fp8_gemm_bf16(s["xq"], s["xs"], s["qkv"][0], s["qkv"][1], s["y_qkv"], t, qkv, h, None)
    # attention itself is not part of the library: its result is a given tensor
    lib.gemb_fp8_quantize(s["attn"], BF16, s["aq"], s["as"], t, a, None)
    lib.gemb_fp8_gemm_bf16(s["aq"], s["as"], s["o"][0], s["o"][1], s["y_o"], t, h, a, None)
    lib.gemb_rmsnorm_residual(s["y_o"], BF16, n1, s["x"], None, s["mid"], BF16, t, h, eps, None, None)
    lib.gemb_nvfp4_rmsnorm_quantize(s["mid"], BF16, n2, s["hq"], s["hs"], t, h, eps, GA, INTERLEAVED, EXACT, None)
    fused, fused_s, gd, ud = s["gate_up"]
    lib.gemb_nvfp4_gemm_gated_quant(s["hq"], s["hs"], fused, fused_s, s["pq"], s["ps"], t, i, h, GA, gd, ud, GP, None)
    dw, ds, dd = s["down"]
    lib.gemb_nvfp4_gemm_bf16(s["pq"], s["ps"], dw, ds, s["y_d"], t, h, i, GP, dd, None)
    lib.gemb_rmsnorm_residual(s["y_d"], BF16, n3, s["mid"], None, s["out"], BF16, t, h, eps, None, None)
    return [s["y_qkv"], s["mid"], s["out"]]


def _prepare_moe(m, c):
    t, h = c["tokens"], c["hidden"]
    w = synthetic_weights(m.dev, seed_of(m), hidden=h, experts=c["experts"], inter=c["inter"], shared_inter=c["shared"])
    layer = MoeLayer(w, t, c["topk"], GA, GP, GP, stages=False)
    layer.fused = True
    if c["router"] == "spec":
        layer.router_scale = (1.0 + m.normal(h, std=0.1)).mul_(float(h) ** 0.5).to(torch.bfloat16).view(torch.int16)
        layer.per_expert_scale = 1.0 + m.normal(c["experts"], std=0.1)
    return {"layer": layer, "x": m.bf16(t, h)}


def seed_of(m):
    return int(torch.randint(0, 1 << 30, (1,), device=m.dev, generator=m.gen).item())


def _run_moe(lib, c, s):
    layer = s["layer"]
    out = layer.forward(s["x"]).view(torch.bfloat16)
    return {"out": out, "ids": layer.ids, "weights": layer.weights, "counts": layer.counts}


def _prepare_head(m, c):
    r, v, h = c["rows"], c["vocab"], c["hidden"]
    w = m.empty(v, h, dtype=torch.int16)
    step = 32768
    for lo in range(0, v, step):
        w[lo:lo + step] = m.bf16(min(step, v - lo), h, std=0.05)
    blocks = m.lib.cdll.gemb_output_head_candidate_blocks()
    return {"w": w, "h": m.normal(r, h), "cand": torch.zeros((r, blocks, 2), dtype=torch.int32, device=m.dev),
            "sel": torch.zeros((r,), dtype=torch.int32, device=m.dev), "blocks": blocks,
            "suppressed": torch.tensor([0, 1, 2, 3], dtype=torch.int32, device=m.dev),
            "logits": m.empty(r, v, dtype=torch.float32)}


def _run_head(lib, c, s):
    r, v, h = c["rows"], c["vocab"], c["hidden"]
    lib.gemb_output_head_candidates(s["w"], s["h"], r, s["suppressed"], 4, None, s["cand"], s["logits"], v, h, None)
    lib.gemb_output_head_argmax(s["cand"], r, s["sel"], None)
    return {"selected": s["sel"], "logits": s["logits"]}


_PREPARE = {"linear": _prepare_linear, "decode": _prepare_decode, "prefill": _prepare_prefill, "moe": _prepare_moe, "head": _prepare_head}
_RUN = {"linear": _run_linear, "decode": _run_decode, "prefill": _run_prefill, "moe": _run_moe, "head": _run_head}


def prepare(case, seed):
    m = _Maker(seed)
    state = _PREPARE[case["family"]](m, case)
    state["case"], state["lib"] = case, m.lib
    return state


def run(state):
    case = state["case"]
    return _RUN[case["family"]](state["lib"], case, state)


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def _fp8(rows, k):
    return rows * k + 2 * rows


def _fp4(rows, k):
    return rows * k * 9 / 16


def _touched_experts(c):
    """Expected number of experts that own at least one of the tokens' assignments, under the router's prior."""
    e, rng = c["experts"], np.random.RandomState(7)
    bias = -1.1 * np.log(np.arange(1, e + 1))
    z = rng.standard_normal((2048, e)) * (0.02 * np.sqrt(c["hidden"])) + (bias - bias.mean())
    picked = np.bincount(np.argpartition(-z, c["topk"] - 1, axis=1)[:, :c["topk"]].ravel(), minlength=e) / 2048.0
    return float(np.sum(1.0 - (1.0 - np.minimum(picked, 1.0)) ** c["tokens"]))


def work(case):
    c, f = case, case["family"]
    if f == "linear":
        t, n, k = c["tokens"], c["rows"], c["k"]
        w = _fp8(n, k) if c["format"] == "fp8" else _fp4(n, k)
        return {"bytes": w + t * k * 2 + t * n * (4 if t == 1 else 2), "flops": 2.0 * t * n * k}
    if f == "decode":
        t, h, a, kv, i = c["tokens"], c["hidden"], c["attention"], c["kv"], c["inter"]
        mlp = (_fp8(2 * i, h) + _fp8(h, i)) if c["mlp"] == "fp8" else _fp4(2 * i, h) + _fp4(h, i)
        acts = t * (a * 4 + (a + 2 * kv) * 4 + h * 8) if c["mlp"] == "nvfp4" else 2 * (2 * h + a + i) + 4 * (a + 2 * kv + 2 * h + 2 * i)
        return {"bytes": c["layers"] * (_fp8(a + 2 * kv, h) + _fp8(h, a) + mlp + acts),
                "flops": 2.0 * t * c["layers"] * ((a + 2 * kv) * h + a * h + 3 * h * i)}
    if f == "prefill":
        t, h, a, qkv, i = c["tokens"], c["hidden"], c["attention"], c["qkv"], c["inter"]
        return {"bytes": _fp8(qkv, h) + _fp8(h, a) + 3 * _fp4(h, i) + 2 * t * (2 * h + a + qkv + h),
                "flops": 2.0 * t * (qkv * h + h * a + 3 * h * i)}
    if f == "moe":
        t, h, e, k, i, s = c["tokens"], c["hidden"], c["experts"], c["topk"], c["inter"], c["shared"]
        return {"bytes": _touched_experts(c) * _fp4(3 * h, i) + _fp4(3 * h, s) + e * h * 4 + t * h * 4 + t * k * 8,
                "flops": 2.0 * t * (e * h + k * 3 * i * h + 3 * s * h)}
    r, v, h = c["rows"], c["vocab"], c["hidden"]
    return {"bytes": v * h * 2.0 + r * h * 4 + r * v * 4, "flops": 2.0 * r * v * h}


def tolerance(case):
    """Single fp32 projections differ by the order of their sums; bf16 outputs by one rounding; in the
    chained decode layers a rounding that falls the other way is a different quantiser code downstream.
    Whole numbers (expert ids, counts, selected tokens) are exact."""
    if case["family"] == "head" or (case["family"] == "linear" and case["tokens"] == 1):
        return {"rel": 1e-5}
    if case["family"] == "decode" and case["mlp"] == "fp8":
        return {"rel": 1e-5}
    return {"rel": 1e-2}
