"""Grouped FP8 GEMMs at the edges of their tiles: experts with chosen row counts (none, around the groups of 8, 16, 32, 128 and
256 rows in which rows are loaded, added to the output and tiled), odd and single K blocks, GEMM2 with one K block and two
(D = 4096) or five (D = 8192) tiles per CTA, five or nine per CTA pair, so that the ring in which a tile's place is handed over
comes round between tiles with full and with padded warps, and GEMM1 with three tiles per CTA or five per pair (I = 2048), so that
activation rows of a fuller tile are left in the stages.  Against the CPU emulation with the bars of the layer's tests (2e-2
relative + 1e-2 absolute)."""
import contextlib

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
RTOL, ATOL = 2e-2, 1e-2
COUNTS = [0, 1, 7, 8, 9, 16, 17, 31, 32, 33, 40, 0, 120, 121, 127, 128, 129, 136, 161, 257, 0]


@pytest.mark.parametrize("option", ["none", "fixed_order", "pow2", "pairs"])
@pytest.mark.parametrize("packed", [False, True])
@pytest.mark.parametrize("D,I", [(768, 384), (4096, 128), (8192, 128), (512, 2048)])
def test_expert_row_counts_at_tile_edges(b200, cuda, D, I, packed, option):
    rng = np.random.default_rng(D + I)
    E, K = len(COUNTS), 2
    owner = np.repeat(np.arange(E), COUNTS).astype(np.int32)
    rng.shuffle(owner)
    T = len(owner)
    ids = np.full((T, K), -1, dtype=np.int32)              # one slot per token, the other one foreign
    ids[np.arange(T), rng.integers(0, K, T)] = owner
    wts = rng.uniform(0.1, 1, (T, K)).astype(np.float32)
    with (oracle.pow2_scales() if option == "pow2" else contextlib.nullcontext()):
        xq, xs = oracle.quant_act(rng.normal(0, 1, (T, D)).astype(np.float32))
        w1q, w1s = oracle.quant_weight(rng.normal(0, D ** -0.5, (E, 2 * I, D)).astype(np.float32))
        w2q, w2s = oracle.quant_weight(rng.normal(0, I ** -0.5, (E, D, I)).astype(np.float32))
        ref = oracle.moe_fp8_experts(xq, xs, w1q, w1s, w2q, w2s, ids, wts, np.arange(T, dtype=np.int32))
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    w1, w2, run = dev(w1q), dev(w2q), b200.moe_fp8_experts
    if packed:
        p1, p2 = torch.empty_like(w1), torch.empty_like(w2)
        b200.moe_fp8_pack_weights(1, w1, p1, E, D, I)
        b200.moe_fp8_pack_weights(2, w2, p2, E, D, I)
        w1, w2, run = p1, p2, b200.moe_fp8_experts_packed
    flags = {"none": 0, "fixed_order": b200.MOE_DETERMINISTIC, "pow2": b200.MOE_POW2_SCALES, "pairs": b200.MOE_CTA_PAIR_TILES}[option]
    cfg = b200.MoeFp8Config(T, E, K, D, I, b200.SCORE_SIGMOID_GROUPED, 1, 1, 1.0, flags)
    out = torch.full((T, D), float("nan"), dtype=torch.float32, device=cuda)
    run(dev(xq), dev(xs), dev(ids), dev(wts), w1, dev(w1s), w2, dev(w2s), out, cfg)
    torch.cuda.synchronize()
    assert b200.device_status() == 0
    got = out.cpu().numpy()
    off = np.abs(got - ref) > ATOL + RTOL * np.abs(ref)
    assert not off.any(), (int(off.sum()), float(np.abs(got - ref).max()), sorted({COUNTS[e] for e in owner[off.any(1)]}))
