"""GPU parity of the MoE path against the CPU restatement: logits, expert ids, routing weights,
counts, offsets and the stable permutation bit for bit; expert outputs within the GEMM gate."""
import numpy as np
import pytest
import torch

from gem16_b200.moe import MoeLayer, MoeWeights
from tests.gemm_util import error_stats
from tests.moe_ref import ffn_oracle, make_layer, moe_layer_oracle
from tests.util import bf16_bits, from_bf16_bits, to_dev, to_np

pytestmark = pytest.mark.gpu

# Relative Frobenius gate of expert and layer outputs (bf16) against the bf16-rounded oracle: the
# path's acceptance rule.  An output differs from the oracle's only where fp32 accumulation order moved
# a value across a bf16 rounding boundary, here or at the bf16 gate/up and product boundaries in the
# middle of the FFN (where one flipped bf16 can also flip an E2M1 code of the down projection's input);
# observed 1.3e-5 on the 4,096-token layer at the model's dimensions.
MOE_GATE = 1e-3


def gpu_route(lib, dev, logits, topk, scale=None, want_probs=False):
    t, e = logits.shape
    ids = torch.full((t, topk), -1, dtype=torch.int32, device=dev)
    w = torch.zeros((t, topk), device=dev)
    probs = torch.zeros((t, e), device=dev) if want_probs else None
    lib.gemb_moe_route(to_dev(logits, dev), None if scale is None else to_dev(scale, dev), ids, w, probs, t, e, topk, None)
    return (to_np(ids), to_np(w)) + ((to_np(probs),) if want_probs else ())


def test_router_kats(lib, dev, orc):
    cases = [np.zeros((3, 128), np.float32)]
    lg = np.full((1, 128), -5.0, np.float32)
    lg[0, [100, 90, 80, 70, 60, 50, 40]] = [7, 6, 5, 4, 3, 2, 1]
    lg[0, [33, 17, 99]] = 0.5
    cases.append(lg)
    lg = np.zeros((1, 128), np.float32); lg[0, 77] = 60.0
    cases.append(lg)
    rng = np.random.default_rng(0)
    cases.append((rng.standard_normal((257, 128)) * 4).astype(np.float32))
    cases.append((rng.standard_normal((64, 256)) * 2).astype(np.float32))
    cases.append(np.round(rng.standard_normal((200, 64)) * 2).astype(np.float32))   # many exact ties
    for lg in cases:
        ids, w, p = gpu_route(lib, dev, lg, 8, want_probs=True)
        oi, ow, op = orc.moe_route(lg, 8, want_probs=True)
        assert np.array_equal(ids, oi)
        assert np.array_equal(w.view(np.uint32), ow.view(np.uint32))
        assert np.array_equal(p.view(np.uint32), op.view(np.uint32))
    assert gpu_route(lib, dev, cases[0], 8)[0].tolist() == [list(range(8))] * 3
    scale = rng.uniform(0.5, 2, 128).astype(np.float32)
    ids, w = gpu_route(lib, dev, cases[3], 8, scale=scale)
    oi, ow = orc.moe_route(cases[3], 8, per_expert_scale=scale)
    assert np.array_equal(ids, oi) and np.array_equal(w.view(np.uint32), ow.view(np.uint32))


# 1-256 / 257-512 / 513-2,048 tokens run the three expert-per-thread kernels, 2,049 and up the tiled
# kernel (8- and 16-token CTAs while those fit the SMs, 32-token CTAs beyond, 64-token CTAs from about 7,000 tokens): every one of them, and the
# sizes the benchmarks run (4,096 and 16,384 tokens x 2,816 x 128), against the oracle bit for bit.
@pytest.mark.parametrize("tokens,hidden,experts", [(1, 64, 32), (77, 2816, 128), (300, 260, 160), (513, 2816, 128),
                                                    (2048, 2816, 128), (2049, 2816, 128), (2051, 260, 160),
                                                    (4096, 2816, 128), (16384, 2816, 128)])
def test_router_logits_bit_exact(lib, dev, orc, tokens, hidden, experts):
    rng = np.random.default_rng(tokens)
    x = bf16_bits(rng.standard_normal((tokens, hidden)).astype(np.float32))
    w = (rng.standard_normal((experts, hidden)) * 0.02).astype(np.float32)
    b = rng.standard_normal(experts).astype(np.float32)
    for bias in (b, None):
        out = torch.zeros((tokens, experts), device=dev)
        lib.gemb_moe_router_logits(to_dev(x, dev), to_dev(w, dev), None if bias is None else to_dev(bias, dev), out,
                                   tokens, hidden, experts, None)
        want = orc.moe_router_logits(x, w, bias)
        assert np.array_equal(to_np(out).view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("tokens,hidden,experts", [(2100, 2816, 128), (333, 264, 160), (70, 2816, 128)])
def test_every_router_kernel_variant_gives_the_same_bits(lib, dev, orc, tokens, hidden, experts):
    """GEMB_TUNE_ROUTER_TILE forces each logits kernel in turn (expert-per-thread, 8 / 16 / 32 / 56 / 64-token tiles):
    all of them against the oracle bit for bit, on a batch with token, expert and K tails."""
    rng = np.random.default_rng(tokens + hidden)
    x = bf16_bits(rng.standard_normal((tokens, hidden)).astype(np.float32))
    w = (rng.standard_normal((experts, hidden)) * 0.02).astype(np.float32)
    b = rng.standard_normal(experts).astype(np.float32)
    want = orc.moe_router_logits(x, w, b)
    xd, wd, bd = to_dev(x, dev), to_dev(w, dev), to_dev(b, dev)
    try:
        for tile in (1, 8, 16, 32, 56, 64):
            lib.gemb_set_tuning(8, tile)
            out = torch.full((tokens, experts), float("nan"), device=dev)
            lib.gemb_moe_router_logits(xd, wd, bd, out, tokens, hidden, experts, None)
            assert np.array_equal(to_np(out).view(np.uint32), want.view(np.uint32)), tile
    finally:
        lib.gemb_set_tuning(8, 0)


@pytest.mark.parametrize("hidden", [4, 36, 128, 260, 544, 2820])
@pytest.mark.parametrize("tokens,experts,shift", [(1, 128, 0), (25, 33, 4), (49, 160, 0), (130, 128, 4)])
def test_router_rings_over_edges(lib, dev, orc, tokens, hidden, experts, shift):
    """Tiles and rings of every logits kernel: K below one tile, with a rest, past the ring's depth; rows of 8-byte alignment only
    (hidden % 8 = 4, or a view that starts `shift` values in); token and expert tails.  Bit for bit, as one chain in ascending k."""
    rng = np.random.default_rng(tokens * hidden)
    x = bf16_bits(rng.standard_normal((tokens, hidden)).astype(np.float32))
    w = (rng.standard_normal((experts, hidden)) * 0.02).astype(np.float32)
    want = orc.moe_router_logits(x, w, None)
    room = torch.zeros(tokens * hidden + 8, dtype=torch.uint16, device=dev)
    xd = room[shift:shift + tokens * hidden]
    xd.copy_(to_dev(x, dev).view(torch.uint16).reshape(-1))
    wd = to_dev(w, dev)
    try:
        for tile in (0, 1, 2, 3, 4, 24, 32, 40, 48, 56, 64):
            lib.gemb_set_tuning(8, tile)
            out = torch.full((tokens, experts), float("nan"), device=dev)
            lib.gemb_moe_router_logits(xd, wd, None, out, tokens, hidden, experts, None)
            assert np.array_equal(to_np(out).view(np.uint32), want.view(np.uint32)), tile
    finally:
        lib.gemb_set_tuning(8, 0)
    lib.gemb_check_device_status()


@pytest.mark.parametrize("tokens", [1, 17, 511, 512, 1023, 4096])
def test_permutation_bit_exact(lib, dev, orc, tokens):
    rng = np.random.default_rng(tokens)
    lg = (rng.standard_normal((tokens, 128)) + rng.standard_normal(128) * 2).astype(np.float32)
    ids, _ = orc.moe_route(lg, 8)
    check_permute(lib, dev, orc, ids, 128)


@pytest.mark.parametrize("assignments,experts", [(1025, 1), (2048, 33), (3 * 1024 + 7, 1024), (17 * 1024 + 1, 128), (147 * 1024, 160),
                                                 (147 * 1024 + 1, 128), (300 * 1024 + 9, 128)])
def test_permutation_over_segments(lib, dev, orc, assignments, experts):
    """Segments of 1,024 assignments: two to the most that one launch places (a CTA per SM), and more (scan and scatter in two launches)."""
    rng = np.random.default_rng(assignments)
    check_permute(lib, dev, orc, rng.integers(0, experts, (assignments, 1)).astype(np.int32), experts)


def test_permutation_zero_hit_and_single_expert(lib, dev, orc):
    check_permute(lib, dev, orc, np.tile(np.arange(8, dtype=np.int32), (700, 1)), 128)      # 120 experts empty
    check_permute(lib, dev, orc, (np.arange(128 * 8, dtype=np.int32).reshape(128, 8)) % 128, 128)


def check_permute(lib, dev, orc, ids, experts):
    t, k = ids.shape
    c = lib.cdll
    counts = torch.full((experts,), -1, dtype=torch.int32, device=dev)
    offsets = torch.full((experts + 1,), -1, dtype=torch.int32, device=dev)
    perm = torch.full((t * k,), -1, dtype=torch.int32, device=dev)
    rows = torch.full((t * k,), -1, dtype=torch.int32, device=dev)
    plan = torch.full((c.gemb_moe_plan_ints(t, experts, k),), -1, dtype=torch.int32, device=dev)
    ws = torch.empty((c.gemb_moe_permute_workspace_bytes(t, experts, k),), dtype=torch.uint8, device=dev)
    lib.gemb_moe_permute(to_dev(ids, dev), counts, offsets, perm, rows, plan, ws, ws.numel(), t, experts, k, None)
    oc, oo, op = orc.moe_permute(ids, experts)
    assert np.array_equal(to_np(counts), oc) and np.array_equal(to_np(offsets), oo) and np.array_equal(to_np(perm), op)
    plan, rows = to_np(plan), to_np(rows)
    # every expert's rows are padded to a multiple of 256; a 128-row tile of padding only is marked -1
    padded = np.concatenate([[0], np.cumsum((oc + 255) // 256 * 256)])
    assert plan[0] == padded[-1] // 128 and plan[1] == padded[-1]
    assert np.array_equal(plan[2:2 + experts + 1], padded)
    info = plan[3 + experts:3 + experts + 2 * plan[0] + 1]       # pairs {expert of tile i, i-th real tile}, then their number
    tile_expert = info[0:2 * plan[0]:2]
    want_tiles = []
    for e in range(experts):
        real = (oc[e] + 127) // 128
        want_tiles += [e] * real + [-1] * ((oc[e] + 255) // 256 * 2 - real)
    assert np.array_equal(tile_expert, np.array(want_tiles, np.int32))
    live_n = info[2 * plan[0]]
    assert live_n == ((oc + 127) // 128).sum()
    assert np.array_equal(info[1:2 * live_n:2], np.nonzero(np.array(want_tiles) >= 0)[0])
    # slot_rows: assignment perm[offsets[e] + j] sits at padded row padded[e] + j
    want_rows = np.empty(t * k, np.int32)
    for e in range(experts):
        want_rows[op[oo[e]:oo[e + 1]]] = padded[e] + np.arange(oc[e])
    assert np.array_equal(rows, want_rows)
    assert plan[0] * 128 <= c.gemb_moe_padded_rows_max(t, experts, k)


def run_layer(lib, dev, orc, tokens, hidden, experts, inter, shared_inter, topk, seed):
    rng = np.random.default_rng(seed)
    p = make_layer(orc, rng, hidden, experts, inter, shared_inter)
    x = bf16_bits(rng.standard_normal((tokens, hidden)).astype(np.float32))
    ga = float(np.float32(2688.0) / np.abs(from_bf16_bits(x)).max())
    ga_dn, ga_sh = 2688.0 / 8.0, 2688.0 / 8.0
    ref = moe_layer_oracle(orc, p, x, topk, ga, ga_dn, ga_sh if shared_inter else None)
    shared = (p["sh_gu"], p["sh_dn"]) if shared_inter else None
    w = MoeWeights(lib, dev, p["router_w"], p["router_bias"], p["gu_packed"], p["gu_scales"], p["gu_div"],
                   p["dn_packed"], p["dn_scales"], p["dn_div"], shared)
    layer = MoeLayer(w, tokens, topk, ga, ga_dn, ga_sh)
    layer._last_x = to_dev(x, dev)
    out = layer.forward(layer._last_x)
    torch.cuda.synchronize()
    lib.gemb_check_device_status()
    # routing: bit exact
    assert np.array_equal(to_np(layer.logits).view(np.uint32), ref["logits"].view(np.uint32))
    assert np.array_equal(to_np(layer.ids), ref["ids"])
    assert np.array_equal(to_np(layer.weights).view(np.uint32), ref["weights"].view(np.uint32))
    assert np.array_equal(to_np(layer.counts), ref["counts"]) and np.array_equal(to_np(layer.perm), ref["perm"])
    # expert outputs per assignment and the combined output: GEMM gate
    rows = to_np(layer.slot_rows)
    y = from_bf16_bits(to_np(layer.y, np.uint16))[rows]
    st = error_stats(y, ref["y_slots"].astype(np.float64))
    assert st["rel_fro"] <= MOE_GATE and st["cos"] > 0.9999, st
    st = error_stats(from_bf16_bits(to_np(out, np.uint16)), from_bf16_bits(ref["out"]).astype(np.float64))
    assert st["rel_fro"] <= MOE_GATE and st["cos"] > 0.9999, st
    print("moe layer errors", st)
    return layer, ref


def test_layer_benchmark_size_routing_in_full(lib, dev, orc):
    """The 4,096-token layer the benchmark runs (26B-A4B dimensions, Zipf router bias): logits, ids,
    weights, counts, offsets, permutation and padded rows compared in full with the oracle; expert and
    combined outputs on 128 sampled tokens (all eight experts of each, plus the shared branch)."""
    from gem16_b200.moe import synthetic_weights
    tokens, hidden, experts, inter, shared_inter, topk = 4096, 2816, 128, 704, 2112, 8
    w = synthetic_weights(dev, 31, hidden, experts, inter, shared_inter, keep_compact=True)
    g = torch.Generator(device=dev)
    g.manual_seed(32)
    x = torch.randn((tokens, hidden), device=dev, generator=g).to(torch.bfloat16).view(torch.int16)
    ga = float(2688.0 / x.view(torch.bfloat16).float().abs().max().item())
    ga_dn = ga_sh = 2688.0 / 8.0
    layer = MoeLayer(w, tokens, topk, ga, ga_dn, ga_sh)
    out = layer.forward(x)
    torch.cuda.synchronize()
    lib.gemb_check_device_status()
    xb = to_np(x, np.uint16)
    logits = orc.moe_router_logits(xb, to_np(w.router_w), to_np(w.router_bias))
    ids, weights = orc.moe_route(logits, topk)
    counts, offsets, perm = orc.moe_permute(ids, experts)
    assert np.array_equal(to_np(layer.logits).view(np.uint32), logits.view(np.uint32))
    assert np.array_equal(to_np(layer.ids), ids)
    assert np.array_equal(to_np(layer.weights).view(np.uint32), weights.view(np.uint32))
    assert np.array_equal(to_np(layer.counts), counts) and np.array_equal(to_np(layer.offsets), offsets)
    assert np.array_equal(to_np(layer.perm), perm)
    padded = np.concatenate([[0], np.cumsum((counts + 255) // 256 * 256)])
    want_rows = np.empty(tokens * topk, np.int32)
    for e in range(experts):
        want_rows[perm[offsets[e]:offsets[e + 1]]] = padded[e] + np.arange(counts[e])
    assert np.array_equal(to_np(layer.slot_rows), want_rows)
    assert counts.max() > 4 * counts.mean()          # the Zipf bias does create the imbalance the config asks for
    # outputs of sampled tokens through the oracle's expert math
    sample = np.sort(np.random.default_rng(33).choice(tokens, 128, replace=False))
    xs_f = from_bf16_bits(xb[sample])
    xq, xsc = orc.nvfp4_quantize(xs_f, ga)
    gu_p, gu_s, dn_p, dn_s = (to_np(t) for t in (w.gu_packed, w.gu_compact, w.dn_packed, w.dn_compact))
    gu_d, dn_d = to_np(w.gu_div), to_np(w.dn_div)
    y_slots = np.zeros((len(sample), topk, hidden), np.float32)
    for e in np.unique(ids[sample]):
        ti, si = np.nonzero(ids[sample] == e)
        y, _, _ = ffn_oracle(orc, xq[ti], xsc[ti], ga, (gu_p[e], gu_s[e], float(gu_d[e])), (dn_p[e], dn_s[e], float(dn_d[e])),
                             ga_dn, inter)
        y_slots[ti, si] = y
    sh = w.shared_compact
    shared, _, _ = ffn_oracle(orc, xq, xsc, ga, sh[0], sh[1], ga_sh, shared_inter)
    want_out = orc.moe_combine(bf16_bits(y_slots), weights[sample], bf16_bits(shared))
    rows = to_np(layer.slot_rows).reshape(tokens, topk)[sample]
    got_y = from_bf16_bits(to_np(layer.y, np.uint16))[rows]
    st = error_stats(got_y.reshape(-1, hidden), y_slots.reshape(-1, hidden).astype(np.float64))
    print("expert outputs", st)
    assert st["rel_fro"] <= MOE_GATE and st["cos"] > 0.9999, st
    st = error_stats(from_bf16_bits(to_np(out, np.uint16))[sample], from_bf16_bits(want_out).astype(np.float64))
    print("layer output", st)
    assert st["rel_fro"] <= MOE_GATE and st["cos"] > 0.9999, st


def test_non_finite_logit_is_recorded_not_followed(lib, dev):
    """A NaN or infinite router logit (MOE_ROUTER_SPEC.md:117-130 wants it visible): the token gets in-range
    ids and zero weights, the other tokens are routed as usual, the permutation works on what it
    is given, and gemb_check_device_status reports kDataLoss once."""
    from gem16_b200.lib import GembError
    rng = np.random.default_rng(3)
    lg = rng.standard_normal((40, 128)).astype(np.float32)
    clean_ids, clean_w = gpu_route(lib, dev, lg, 8)
    lib.gemb_check_device_status()
    lg[7, 100] = np.nan
    lg[21, 3] = np.inf
    ids, w = gpu_route(lib, dev, lg, 8)
    with pytest.raises(GembError) as err:
        lib.gemb_check_device_status()
    assert err.value.status_name == "kDataLoss"
    lib.gemb_check_device_status()                     # cleared once read
    assert ids.min() >= 0 and ids.max() < 128
    for t in (7, 21):
        assert ids[t].tolist() == list(range(8)) and not w[t].any()
    keep = np.setdiff1d(np.arange(40), [7, 21])
    assert np.array_equal(ids[keep], clean_ids[keep]) and np.array_equal(w[keep], clean_w[keep])


def test_out_of_range_expert_id_is_clamped_and_recorded(lib, dev, orc):
    from gem16_b200.lib import GembError
    ids = np.tile(np.arange(8, dtype=np.int32), (50, 1))
    ids[3, 2] = 128          # one past the last expert
    ids[9, 0] = -5
    ids[40, 7] = 0x7FFFFFFF
    clamped = np.where((ids < 0) | (ids >= 128), 127, ids).astype(np.int32)
    t, k = ids.shape
    c = lib.cdll
    i32 = dict(dtype=torch.int32, device=dev)
    counts, offsets = torch.zeros((128,), **i32), torch.zeros((129,), **i32)
    perm, rows = torch.full((t * k,), -1, **i32), torch.full((t * k,), -1, **i32)
    plan = torch.zeros((c.gemb_moe_plan_ints(t, 128, k),), **i32)
    ws = torch.empty((c.gemb_moe_permute_workspace_bytes(t, 128, k),), dtype=torch.uint8, device=dev)
    lib.gemb_moe_permute(to_dev(ids, dev), counts, offsets, perm, rows, plan, ws, ws.numel(), t, 128, k, None)
    torch.cuda.synchronize()
    with pytest.raises(GembError) as err:
        lib.gemb_check_device_status()
    assert err.value.status_name == "kDataLoss"
    oc, oo, op = orc.moe_permute(clamped, 128)
    assert np.array_equal(to_np(counts), oc) and np.array_equal(to_np(offsets), oo) and np.array_equal(to_np(perm), op)
    assert to_np(rows).min() >= 0 and to_np(rows).max() < c.gemb_moe_padded_rows_max(t, 128, k)


def test_layer_small(lib, dev, orc):
    run_layer(lib, dev, orc, tokens=77, hidden=256, experts=32, inter=128, shared_inter=128, topk=4, seed=5)


def test_layer_real_dims(lib, dev, orc):
    # 26B-A4B dimensions (hidden 2816, 128 experts x 704, top-8, shared 2112) at a decode-size batch
    layer, ref = run_layer(lib, dev, orc, tokens=64, hidden=2816, experts=128, inter=704, shared_inter=2112, topk=8, seed=6)
    # repeated-run identity of routing records and outputs (deterministic mode is the only mode)
    first = [t.clone() for t in (layer.ids, layer.weights, layer.perm, layer.out)]
    layer.forward(layer._last_x)
    torch.cuda.synchronize()
    for a, b in zip(first, (layer.ids, layer.weights, layer.perm, layer.out)):
        assert torch.equal(a, b)
    assert int(to_np(layer.counts).sum()) == 64 * 8


def test_fused_gated_epilogue_is_byte_identical(lib, dev, orc):
    # One kernel (gate/up GEMM + GELU + requantisation) against the three-launch form, on the
    # expert path (grouped, K = hidden) and the shared branch (rows not a multiple of 128).
    rng = np.random.default_rng(21)
    tokens, hidden, experts, inter, shared_inter, topk = 300, 2816, 128, 704, 2112, 8
    from gem16_b200.moe import synthetic_weights
    w = synthetic_weights(dev, 5, hidden, experts, inter, shared_inter)
    x = to_dev(bf16_bits(rng.standard_normal((tokens, hidden)).astype(np.float32)), dev)
    layer = MoeLayer(w, tokens, topk, 700.0, 336.0, 336.0)
    results = []
    for fused in (False, True):
        layer.fused = fused
        for t in (layer.p_packed, layer.p_scales, layer.s_p_packed, layer.s_p_scales):
            t.zero_()
        out = layer.forward_stages(x).clone()
        torch.cuda.synchronize()
        lib.gemb_check_device_status()
        rows = layer.slot_rows.long()
        blocks = torch.arange(inter // 16, device=dev)
        # scales of the valid rows only (padding rows of the padded space hold garbage by design)
        c_pad = (inter // 16 + 3) // 4 * 4
        off = ((rows[:, None] // 128) * (c_pad // 4) + blocks[None, :] // 4) * 512 + (rows[:, None] % 32) * 16 \
            + ((rows[:, None] % 128) // 32) * 4 + blocks[None, :] % 4
        results.append((layer.p_packed[rows].clone(), layer.p_scales[off].clone(), layer.s_p_packed.clone(),
                        layer.s_p_scales.clone(), layer.y[rows].clone(), out))
    for a, b in zip(*results):
        assert torch.equal(a, b)


@pytest.mark.parametrize("fused", [False, True])
def test_library_layer_call_equals_the_stage_launches(lib, dev, fused):
    """gemb_moe_layer_forward (the launch sequence inside the library, workspace filled with 0xFF
    beforehand, shared branch forked onto a second stream) against the same operators launched one
    by one: identical records and identical output bytes, with and without the fused GELU epilogue,
    and the same again without a second stream."""
    from gem16_b200.moe import synthetic_weights
    tokens, topk = 333, 8
    w = synthetic_weights(dev, 9)
    g = torch.Generator(device=dev)
    g.manual_seed(10)
    x = torch.randn((tokens, 2816), device=dev, generator=g).to(torch.bfloat16).view(torch.int16)
    a, b = MoeLayer(w, tokens, topk, 650.0, 336.0, 336.0), MoeLayer(w, tokens, topk, 650.0, 336.0, 336.0)
    a.fused = b.fused = fused
    want = a.forward_stages(x).clone()
    got = b.forward(x).clone()
    torch.cuda.synchronize()
    lib.gemb_check_device_status()
    for name in ("logits", "ids", "weights", "counts", "offsets", "perm", "slot_rows"):
        assert torch.equal(getattr(a, name), getattr(b, name)), name
    rows = a.slot_rows.long()
    assert torch.equal(a.y[rows], b.y[rows]) and torch.equal(want, got)
    # everything on one stream
    desc = w.c_struct(topk, 650.0, 336.0, 336.0, fused=fused)
    out = torch.zeros_like(got)
    lib.gemb_moe_layer_forward(desc, x, out, tokens, b.c_base, b.c_workspace.numel() - 256, None, None, None, None)
    torch.cuda.synchronize()
    assert torch.equal(out, got)
    # grouped GEMMs forced onto CTA pairs (256-row units, the odd CTA of a unit often on padding only) and onto
    # single CTAs (the automatic choice at this size): the same bytes
    try:
        for mode in (2, 1):
            lib.gemb_set_tuning(5, mode)
            out.zero_()
            lib.gemb_moe_layer_forward(desc, x, out, tokens, b.c_base, b.c_workspace.numel() - 256, None, None, None, None)
            torch.cuda.synchronize()
            lib.gemb_check_device_status()
            assert torch.equal(out, got), mode
    finally:
        lib.gemb_set_tuning(5, 0)
    # too small a workspace, a missing weight: rejected before anything runs
    from gem16_b200.lib import GembError
    with pytest.raises(GembError):
        lib.gemb_moe_layer_forward(desc, x, out, tokens, b.c_base, 1024, None, None, None, None)
    desc.down.packed_weight = None
    with pytest.raises(GembError):
        lib.gemb_moe_layer_forward(desc, x, out, tokens, b.c_base, b.c_workspace.numel() - 256, None, None, None, None)


@pytest.mark.parametrize("tokens,hidden,topk,offset", [(1, 8, 1, 0), (37, 2816, 8, 0), (37, 2816, 8, 1), (300, 136, 5, 0), (65, 264, 32, 0),
                                                       (9, 1032, 6, 0), (130, 72, 4, 3)])
@pytest.mark.parametrize("by_row", [True, False])
def test_combine_forms(lib, dev, orc, tokens, hidden, topk, offset, by_row):
    """Four slots to a load and one by one (top-k no multiple of four, records off a 16-byte boundary, rows in assignment order),
    with and without the shared branch: the oracle's fma chain, bit for bit."""
    rng = np.random.default_rng(tokens * 100 + topk)
    n = tokens * topk
    rows = n + 77 if by_row else n
    y = bf16_bits(rng.standard_normal((rows, hidden)).astype(np.float32))
    slots = rng.permutation(rows)[:n].astype(np.int32) if by_row else np.arange(n, dtype=np.int32)
    weights = rng.random((tokens, topk)).astype(np.float32)
    shared = bf16_bits(rng.standard_normal((tokens, hidden)).astype(np.float32))

    def shifted(a):
        buf = torch.zeros((n + 4,), dtype=torch.float32 if a.dtype == np.float32 else torch.int32, device=dev)
        buf[offset:offset + n] = to_dev(a.reshape(-1), dev)
        return buf[offset:offset + n]

    d_slots, d_weights = (shifted(slots) if by_row else None), shifted(weights)
    for sh in (shared, None):
        out = torch.full((tokens, hidden), 0x7FC0, dtype=torch.int16, device=dev)
        lib.gemb_moe_combine(to_dev(y, dev), d_slots, d_weights, None if sh is None else to_dev(sh, dev), out, tokens, hidden, topk, None)
        want = orc.moe_combine(y[slots].reshape(tokens, topk, hidden), weights, sh)
        assert np.array_equal(to_np(out, np.uint16), np.asarray(want).view(np.uint16).reshape(tokens, hidden))


def test_shared_branch_bits_depend_on_the_token_alone(lib, dev):
    """A layer whose shared branch has a long K and few tiles: the first 77 of 300 tokens by themselves (an expert-parallel
    rank holds a part of the tokens) and with the others, through the fused epilogue and without it, give the same bytes."""
    from gem16_b200.moe import synthetic_weights
    w = synthetic_weights(dev, 3, hidden=4096, experts=32, inter=64, shared_inter=4096)
    g = torch.Generator(device=dev)
    g.manual_seed(4)
    x = torch.randn((300, 4096), device=dev, generator=g).to(torch.bfloat16).view(torch.int16)
    outs = []
    for tokens in (300, 77):
        for fused in (True, False):
            layer = MoeLayer(w, tokens, 4, 650.0, 336.0, 336.0)
            layer.fused = fused
            outs.append(layer.forward(x[:tokens].contiguous())[:77].clone())
    torch.cuda.synchronize()
    lib.gemb_check_device_status()
    for o in outs[1:]:
        assert torch.equal(o, outs[0])


def test_router_specification_mode(lib, dev, orc):
    """The router as docs/plans/gemma4-26b/specs/MOE_ROUTER_SPEC.md:3-13,41-63 writes it: r =
    rmsnorm_noweight(x) * scale * hidden^-1/2, logits = W r (no bias), softmax, top-8, renormalise,
    times per_expert_scale -- the transformed input, ids and weights bit for bit against the oracle,
    alone and through the layer call."""
    from gem16_b200.moe import synthetic_weights
    rng = np.random.default_rng(12)
    tokens, hidden, experts, topk = 200, 2816, 128, 8
    x = bf16_bits((rng.standard_normal((tokens, hidden)) * 3).astype(np.float32))
    scale = bf16_bits((1.0 + 0.3 * rng.standard_normal(hidden)).astype(np.float32))
    pes = rng.uniform(0.5, 2.0, experts).astype(np.float32)
    want_r = orc.moe_router_input(x, scale, 1e-6)
    got_r = torch.zeros((tokens, hidden), dtype=torch.int16, device=dev)
    lib.gemb_moe_router_input(to_dev(x, dev), to_dev(scale, dev), got_r, tokens, hidden, 1e-6, None)
    assert np.array_equal(to_np(got_r, np.uint16), want_r)
    w = synthetic_weights(dev, 13, zipf=False)
    layer = MoeLayer(w, tokens, topk, 650.0, 336.0, 336.0, stages=False)
    layer.router_scale, layer.per_expert_scale = to_dev(scale, dev), to_dev(pes, dev)
    layer.forward(to_dev(x, dev))
    torch.cuda.synchronize()
    lib.gemb_check_device_status()
    logits = orc.moe_router_logits(want_r, to_np(w.router_w), None)
    ids, weights = orc.moe_route(logits, topk, per_expert_scale=pes)
    assert np.array_equal(to_np(layer.logits).view(np.uint32), logits.view(np.uint32))
    assert np.array_equal(to_np(layer.ids), ids)
    assert np.array_equal(to_np(layer.weights).view(np.uint32), weights.view(np.uint32))


@pytest.mark.parametrize("tokens,hidden,offset", [(1, 8, 0), (9, 520, 0), (13, 2816, 1), (3, 12288, 0), (2, 12296, 0)])
def test_router_input_rows_in_shared_memory(lib, dev, orc, tokens, hidden, offset):
    """Partial last CTA, rows that end inside a 1,024-byte piece, an output without 16-byte alignment, and the
    row lengths on both sides of the shared-memory limit: the bits of the oracle's serial chain."""
    rng = np.random.default_rng(tokens + hidden)
    x = bf16_bits(rng.standard_normal((tokens, hidden)).astype(np.float32))
    scale = bf16_bits(1.0 + 0.1 * rng.standard_normal(hidden).astype(np.float32))
    got = torch.zeros((tokens * hidden + offset,), dtype=torch.int16, device=dev)
    lib.gemb_moe_router_input(to_dev(x, dev), to_dev(scale, dev), got[offset:], tokens, hidden, 1e-6, None)
    want = orc.moe_router_input(x, scale, 1e-6)
    assert np.array_equal(to_np(got[offset:]).view(np.uint16).reshape(tokens, hidden), want)


@pytest.mark.parametrize("tokens", [192, 3001])
def test_layer_bytes_do_not_change_between_calls(lib, dev, tokens):
    """The GEMM's operand and scale rings under two streams and changing inputs: same input, same bytes, every call."""
    from gem16_b200.moe import synthetic_weights
    layer = MoeLayer(synthetic_weights(dev, 7), tokens, 8, 600.0, 336.0, 336.0, stages=False)
    layer.fused = True
    g = torch.Generator(device=dev).manual_seed(tokens)
    x, other = (torch.randn((tokens, 2816), device=dev, generator=g).bfloat16().view(torch.int16) for _ in range(2))
    want = layer.forward(x).clone()
    outs = []
    for _ in range(100 if tokens < 1000 else 20):
        layer.forward(other)
        outs.append(layer.forward(x).clone())
    assert all(torch.equal(o, want) for o in outs)


@pytest.mark.parametrize("tile", [1, 2, 3, 4, 24, 40, 48])
@pytest.mark.parametrize("tokens,hidden,experts,offset", [(131, 132, 160, 0), (97, 260, 32, 1), (9, 2816, 128, 0), (1, 4, 32, 0)])
def test_router_shapes_at_their_edges(lib, dev, orc, tile, tokens, hidden, experts, offset):
    """Token, expert and K remainders of the shapes the sweep above does not force; rows only 8-byte aligned."""
    rng = np.random.default_rng(tokens + tile)
    x = bf16_bits(rng.standard_normal((tokens, hidden)).astype(np.float32))
    w = (rng.standard_normal((experts, hidden)) * 0.02).astype(np.float32)
    b = rng.standard_normal(experts).astype(np.float32)
    xd = torch.zeros(tokens * hidden + 4, dtype=torch.int16, device=dev)[4 * offset:][:tokens * hidden].view(tokens, hidden)
    xd.copy_(to_dev(x, dev).view(torch.int16))
    out = torch.full((tokens, experts), float("nan"), device=dev)
    try:
        lib.gemb_set_tuning(8, tile)
        lib.gemb_moe_router_logits(xd, to_dev(w, dev), to_dev(b, dev), out, tokens, hidden, experts, None)
    finally:
        lib.gemb_set_tuning(8, 0)
    assert np.array_equal(to_np(out).view(np.uint32), orc.moe_router_logits(x, w, b).view(np.uint32))


def test_plan_lists_the_rows_of_every_tile(lib, dev):
    """Behind the number of real tiles: rows of each 128-row tile that hold assignments (0, partial, full)."""
    experts, t, k = 32, 300, 2
    ids = torch.zeros((t, k), dtype=torch.int32, device=dev)      # expert 0: 300 rows, expert 5: 33, the rest on 31
    ids[:33, 1], ids[33:, 1] = 5, 31
    c = lib.cdll
    plan = torch.full((c.gemb_moe_plan_ints(t, experts, k),), -1, dtype=torch.int32, device=dev)
    counts, offsets = torch.zeros(experts, dtype=torch.int32, device=dev), torch.zeros(experts + 1, dtype=torch.int32, device=dev)
    perm, rows = (torch.zeros(t * k, dtype=torch.int32, device=dev) for _ in range(2))
    ws = torch.empty((c.gemb_moe_permute_workspace_bytes(t, experts, k),), dtype=torch.uint8, device=dev)
    lib.gemb_moe_permute(ids, counts, offsets, perm, rows, plan, ws, ws.numel(), t, experts, k, None)
    p = to_np(plan)
    assert p[3 + experts + 2 * p[0] + 1:][:p[0]].tolist() == [128, 128, 44, 0, 33, 0, 128, 128, 11, 0]
