"""The FP8 layer as a captured CUDA graph, replayed on inputs that changed since the capture: quantiser, router, sort and both
grouped GEMMs are launched programmatically, each behind the kernel in front of it, and the graph holds those dependencies (and the
memsets between them).  Both sort paths (T K up to 2048 pairs and above), every combine and tile shape.  Against the CPU emulation with
the bars of the layer's tests (2e-2 relative + 1e-2 absolute); with the fixed-order combine the replay gives the bits of a plain call."""
import contextlib

import numpy as np
import pytest
import torch

import oracle

pytestmark = pytest.mark.gpu
RTOL, ATOL = 2e-2, 1e-2
E, K, D, I = 16, 8, 512, 256


@pytest.mark.parametrize("option", ["none", "fixed_order", "pow2", "pairs"])
@pytest.mark.parametrize("T", [1, 40, 300])
def test_captured_layer_follows_its_inputs(b200, cuda, T, option):
    rng = np.random.default_rng(T)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(cuda)
    pow2 = option == "pow2"
    scales = oracle.pow2_scales if pow2 else contextlib.nullcontext
    wg = rng.normal(0, D ** -0.5, (E, D)).astype(np.float32)
    bias = rng.normal(0, 0.01, E).astype(np.float32)
    with scales():
        w1q, w1s = oracle.quant_weight(rng.normal(0, D ** -0.5, (E, 2 * I, D)).astype(np.float32))
        w2q, w2s = oracle.quant_weight(rng.normal(0, I ** -0.5, (E, D, I)).astype(np.float32))
    weights = [dev(a) for a in (wg, bias, w1q, w1s, w2q, w2s)]
    flags = {"none": 0, "fixed_order": b200.MOE_DETERMINISTIC, "pow2": b200.MOE_POW2_SCALES, "pairs": b200.MOE_CTA_PAIR_TILES}[option]
    cfg = b200.MoeFp8Config(T, E, K, D, I, b200.SCORE_SIGMOID_GROUPED, 4, 2, 2.5, flags)
    x = torch.zeros((T, D), device=cuda)
    xq = torch.empty((T, D), dtype=torch.uint8, device=cuda)
    xs = torch.empty((T, D // 128), device=cuda)
    out = torch.empty((T, D), device=cuda)

    def layer(y):
        b200.quant_act_1x128(x, xq, xs, pow2=pow2)
        b200.moe_fp8_forward(xq, xs, *weights, y, cfg)

    layer(out)                                   # the workspace has its size before the capture
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        layer(out)
    for _ in range(3):
        xh = rng.normal(0, 1, (T, D)).astype(np.float32)
        x.copy_(dev(xh))
        out.fill_(float("nan"))
        graph.replay()
        graph.replay()                           # back to back: the second clears and sorts behind the first
        torch.cuda.synchronize()
        assert b200.device_status() == 0
        got = out.cpu().numpy()
        with scales():
            hq, hs = oracle.quant_act(xh)
            ids, wts = oracle.route_grouped(hq, hs, wg, bias, K, 4, 2, 2.5)
            ref = oracle.moe_fp8_experts(hq, hs, w1q, w1s, w2q, w2s, ids, wts, np.arange(T, dtype=np.int32))
        assert not (np.abs(got - ref) > ATOL + RTOL * np.abs(ref)).any()
        if option == "fixed_order":
            plain = torch.empty_like(out)
            layer(plain)
            assert torch.equal(plain, out)
