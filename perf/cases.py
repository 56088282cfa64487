"""Workloads of the two inference layers, called as a serving program calls them.

Every case is a dict of plain values.  ``prepare`` builds what such a program holds before the call (inputs,
weights, caches), ``run`` makes one pass through the package's public entry points, ``work`` counts the bytes and
operations the pass cannot do without, ``tolerance`` says how far another correct implementation may be off.

Kinds of case:
  moe_f32   moe_forward on fp32 tensors (softmax router), the sizes of the fp32 tests and benchmark
  dsa_f32   dsa_forward on fp32 tensors
  moe_fp8   the FP8 block-scale layer: activations quantised to 1x128 blocks, then MoeFp8Layer.forward (router,
            grouped GEMMs, combine); `layout` packed / rows (pre-tiled weights or row-major ones), `option` none /
            pow2 (power-of-two scales) / fixed_order (bit-reproducible combine)
  experts   the owner side of the expert-parallel layer: rows with their slots given, foreign slots -1
  dsa_bf16  sparse MLA decode on a bf16 cache; `ids` flat (physical rows) or paged (positions + block table +
            valid lengths)

``exact`` states the result of a pass in 64-bit torch arithmetic, for measuring how far an implementation is off.
"""
import importlib
import math

import torch

b200 = importlib.import_module("llm-sys-project_b200")


# ---------------------------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------------------------
def _fp8(T, layout="packed", option="none", E=256, K=8, D=7168, I=2048):
    return dict(kind="moe_fp8", T=T, E=E, K=K, D=D, I=I, layout=layout, option=option)


def listed():
    return [
        # the fp32 layer at the parity shape: five small launches, nothing but latency
        dict(name="moe_f32_t32", kind="moe_f32", T=32, E=8, K=2, D=128, I=256),
        # the largest fp32 shape of the benchmark driver
        dict(name="moe_f32_t128", kind="moe_f32", T=128, E=16, K=2, D=512, I=1024),
        # small fp32 decode: a page table of 16 pages per sequence, 256 selected tokens
        dict(name="dsa_f32_q4", kind="dsa_f32", Q=4, H=16, Dc=512, Dp=64, S=256, N=4096),
        # one token: the latency of a single user's decode step
        dict(_fp8(1), name="fp8_t1"),
        # a small decode batch: about a third of the experts active, one or two rows each
        dict(_fp8(16), name="fp8_t16"),
        # an odd batch on the row-major weights a program has that never pre-tiled them
        dict(_fp8(333, layout="rows"), name="fp8_t333_rows"),
        # a chunk of a prefill with the bit-reproducible combine
        dict(_fp8(1024, option="fixed_order"), name="fp8_t1024_fixed_order"),
        # a full prefill step, the benchmark's headline
        dict(_fp8(4096), name="fp8_t4096"),
        # the same with power-of-two scales (UE8M0 checkpoints)
        dict(_fp8(4096, option="pow2"), name="fp8_t4096_pow2"),
        # one GPU of eight under expert parallelism: 32 local experts, about a thousand rows each
        dict(name="experts_r16384", kind="experts", R=16384, E=32, K=8, D=7168, I=2048, layout="packed"),
        # a decode step of 64 sequences with 2048 selected tokens each
        dict(name="dsa_bf16_q64", kind="dsa_bf16", Q=64, H=128, S=2048, ids="flat", seq_min=8192, seq_max=131072),
        # a small decode batch through the block table, some sequences shorter than the selection
        dict(name="dsa_bf16_q5_paged", kind="dsa_bf16", Q=5, H=128, S=2048, ids="paged", seq_min=700, seq_max=16384),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["moe_fp8", "dsa_bf16", "experts", "moe_f32", "dsa_f32"], [5, 2.5, 1, 1, 1])[0]
    if kind == "moe_fp8":
        return _fp8(_log(rng, 1, 4096), layout=rng.choice(["packed", "packed", "rows"]),
                    option=rng.choice(["none", "none", "none", "pow2", "fixed_order"]),
                    E=rng.choice([32, 64, 128, 160, 256, 256]), K=rng.choice([4, 6, 8, 8]),
                    D=256 * rng.randint(8, 28), I=128 * rng.randint(4, 16))
    if kind == "experts":
        return dict(kind="experts", R=_log(rng, 64, 16384), E=rng.choice([16, 32, 64]), K=8, D=256 * rng.randint(8, 28),
                    I=128 * rng.randint(4, 16), layout=rng.choice(["packed", "rows"]))
    if kind == "dsa_bf16":
        S = rng.choice([128 * rng.randint(2, 16), 128 * rng.randint(2, 16), 64 * rng.randint(3, 32),
                        32 * rng.randint(3, 64)])
        return dict(kind="dsa_bf16", Q=_log(rng, 1, 64), H=rng.choice([16, 64, 128, 128]), S=S,
                    ids=rng.choice(["flat", "paged"]), seq_min=S, seq_max=_log(rng, 2 * S, 131072))
    if kind == "moe_f32":
        return dict(kind="moe_f32", T=_log(rng, 16, 128), E=rng.choice([4, 8, 16]), K=rng.choice([2, 4]),
                    D=rng.randint(16, 128) * 4, I=rng.randint(32, 256) * 4)
    return dict(kind="dsa_f32", Q=_log(rng, 1, 16), H=rng.choice([4, 8, 16]), Dc=rng.choice([64, 128, 256, 512]),
                Dp=rng.choice([16, 32, 64]), S=rng.randint(32, 1024), N=rng.choice([1024, 4096, 8192]))


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
DEV = "cuda"
N_GROUP, TOPK_GROUP, ROUTED_SCALE = 8, 4, 2.5


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _normal(shape, seed, sigma, dtype=torch.float32):
    t = torch.empty(shape, dtype=dtype, device=DEV)
    return b200.fill_normal_(t, seed, sigma)


def _fp8_weights(c, seed):
    """Weights of E experts ~ N(0, 0.02) in 128x128 blocks, router weights with unit-variance logits."""
    E, K, D, I = c["E"], c["K"], c["D"], c["I"]
    pow2 = c.get("option") == "pow2"
    w1q = torch.empty((E, 2 * I, D), dtype=torch.uint8, device=DEV)
    w1s = torch.empty((E, 2 * I // 128, D // 128), dtype=torch.float32, device=DEV)
    w2q = torch.empty((E, D, I), dtype=torch.uint8, device=DEV)
    w2s = torch.empty((E, D // 128, I // 128), dtype=torch.float32, device=DEV)
    b200.fill_normal_fp8_w128_(w1q, w1s, seed * 16 + 1, 0.02, pow2=pow2)
    b200.fill_normal_fp8_w128_(w2q, w2s, seed * 16 + 2, 0.02, pow2=pow2)
    gate_w = _normal((E, D), seed * 16 + 3, D ** -0.5)
    bias = _normal((E,), seed * 16 + 4, 0.01)
    return gate_w, bias, w1q, w1s, w2q, w2s


def _fp8_layer(c, seed):
    """The layer object a serving program keeps."""
    gate_w, bias, w1q, w1s, w2q, w2s = _fp8_weights(c, seed)
    flags = {"pow2": b200.MOE_POW2_SCALES, "fixed_order": b200.MOE_DETERMINISTIC}.get(c.get("option"), 0)
    layer = b200.MoeFp8Layer(gate_w, bias, w1q, w1s, w2q, w2s, c["K"], b200.SCORE_SIGMOID_GROUPED, N_GROUP, TOPK_GROUP,
                             ROUTED_SCALE, flags=flags)
    if c["layout"] == "packed":
        layer.pack(free_unpacked=True)
    return layer


def _decode_ids(c, seed):
    """Sequence lengths, the block table of a cache whose pages are handed out at random, and each query's
    selected positions (uniform, no replacement, unsorted; -1 behind the end of a short sequence)."""
    Q, S, page = c["Q"], c["S"], 64
    g = _gen(seed)
    seq = torch.randint(c["seq_min"], c["seq_max"] + 1, (Q,), generator=g, device=DEV)
    blocks = (seq + page - 1) // page
    total = int(blocks.sum())
    perm = torch.randperm(total, generator=g, device=DEV)
    start = torch.cumsum(blocks, 0) - blocks
    max_blocks = int(blocks.max())
    j = torch.arange(max_blocks, device=DEV)
    at = (start[:, None] + j).clamp(max=total - 1)
    table = torch.where(j < blocks[:, None], perm[at], torch.full_like(at, -1)).to(torch.int32)
    pos = torch.full((Q, S), -1, dtype=torch.int64, device=DEV)
    for q, n in enumerate(seq.tolist()):
        m = min(n, S)
        pos[q, :m] = torch.randperm(n, generator=g, device=DEV)[:m]
    return seq.clamp(max=S).to(torch.int32), table, pos, total * page


def prepare(case, seed):
    c = case
    kind = c["kind"]
    if kind == "moe_f32":
        T, E, K, D, I = c["T"], c["E"], c["K"], c["D"], c["I"]
        return dict(kind=kind, x=_normal((T, D), seed * 16, 1.0), wg=_normal((E, D), seed * 16 + 1, D ** -0.5),
                    w1=_normal((E, 2 * I, D), seed * 16 + 2, D ** -0.5), w2=_normal((E, D, I), seed * 16 + 3, I ** -0.5),
                    out=torch.empty((T, D), dtype=torch.float32, device=DEV), cfg=b200.MoeConfig(T, E, K, D, I))
    if kind == "dsa_f32":
        Q, H, Dc, Dp, S, N = c["Q"], c["H"], c["Dc"], c["Dp"], c["S"], c["N"]
        g = _gen(seed)
        idx = torch.stack([torch.randperm(N, generator=g, device=DEV)[:S] for _ in range(Q)]).to(torch.int32)
        return dict(kind=kind, qn=_normal((Q, H, Dc), seed * 16, 1.0), qp=_normal((Q, H, Dp), seed * 16 + 1, 1.0),
                    kc=_normal((N, Dc), seed * 16 + 2, 1.0), kp=_normal((N, Dp), seed * 16 + 3, 1.0),
                    v=_normal((N, Dc), seed * 16 + 4, 1.0), idx=idx,
                    out=torch.empty((Q, H, Dc), dtype=torch.float32, device=DEV),
                    cfg=b200.DsaConfig(Q, H, Dc, Dp, S, 64, N))
    if kind == "moe_fp8":
        T, D = c["T"], c["D"]
        return dict(kind=kind, layer=_fp8_layer(c, seed), x=_normal((T, D), seed * 16 + 5, 1.0),
                    xq=torch.empty((T, D), dtype=torch.uint8, device=DEV),
                    xs=torch.empty((T, D // 128), dtype=torch.float32, device=DEV),
                    out=torch.empty((T, D), dtype=torch.float32, device=DEV), pow2=c["option"] == "pow2")
    if kind == "experts":
        R, E, K, D = c["R"], c["E"], c["K"], c["D"]
        g = _gen(seed)
        x = _normal((R, D), seed * 16 + 5, 1.0)
        xq = torch.empty((R, D), dtype=torch.uint8, device=DEV)
        xs = torch.empty((R, D // 128), dtype=torch.float32, device=DEV)
        b200.quant_act_1x128(x, xq, xs)
        # one to four local experts per row (two on average), some experts busier than others
        score = torch.rand((R, E), generator=g, device=DEV) + 0.3 * torch.rand((E,), generator=g, device=DEV)
        top = score.topk(min(4, E), dim=1).indices.to(torch.int32)
        used = 1 + (torch.rand((R, 3), generator=g, device=DEV) < 1.0 / 3).sum(1)
        rid = torch.full((R, K), -1, dtype=torch.int32, device=DEV)
        rid[:, :top.shape[1]] = torch.where(torch.arange(top.shape[1], device=DEV) < used[:, None], top, torch.full_like(top, -1))
        rw = torch.where(rid >= 0, 0.1 + 0.5 * torch.rand((R, K), generator=g, device=DEV), torch.zeros((R, K), device=DEV))
        return dict(kind=kind, layer=_fp8_layer(c, seed), xq=xq, xs=xs, rid=rid, rw=rw)
    Q, H, S = c["Q"], c["H"], c["S"]
    valid, table, pos, N = _decode_ids(c, seed)
    kc, kp, v = (_normal((N, d), seed * 16 + i, 0.5, torch.bfloat16) for i, d in enumerate((512, 64, 512)))
    s = dict(kind=kind, ids=c["ids"], qn=_normal((Q, H, 512), seed * 16 + 3, 1.0, torch.bfloat16),
             qp=_normal((Q, H, 64), seed * 16 + 4, 1.0, torch.bfloat16),
             out=torch.empty((Q, H, 512), dtype=torch.float32, device=DEV))
    if c["ids"] == "flat":
        page = table.gather(1, (pos.clamp(min=0) // 64)).to(torch.int64)
        s["idx"] = torch.where(pos >= 0, page * 64 + pos % 64, pos).to(torch.int32)
        s["layer"] = b200.DsaDecodeLayer(kc, kp, v, 64)
    else:
        s.update(kc=kc, kp=kp, v=v, pos=pos.to(torch.int32), table=table, valid=valid, cfg=b200.DsaConfig(Q, H, 512, 64, S, 64, N))
    return s


# ---------------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "moe_f32":
        b200.moe_forward(s["x"], s["wg"], s["w1"], s["w2"], s["out"], s["cfg"])
        return s["out"]
    if kind == "dsa_f32":
        b200.dsa_forward(s["qn"], s["qp"], s["kc"], s["kp"], s["v"], s["idx"], s["out"], s["cfg"])
        return s["out"]
    if kind == "moe_fp8":
        b200.quant_act_1x128(s["x"], s["xq"], s["xs"], pow2=s["pow2"])
        return s["xq"], s["xs"], s["layer"].forward(s["xq"], s["xs"], s["out"])
    if kind == "experts":
        return s["layer"].local_experts(s["xq"], s["xs"], s["rid"], s["rw"])
    if s["ids"] == "flat":
        return s["layer"].forward(s["qn"], s["qp"], s["idx"], s["out"])
    b200.dsa_forward_bf16_paged(s["qn"], s["qp"], s["kc"], s["kp"], s["v"], s["pos"], s["table"], s["out"], s["cfg"],
                                valid_len=s["valid"])
    return s["out"]


# ---------------------------------------------------------------------------------------------
# the same results in 64 bits
# ---------------------------------------------------------------------------------------------
def _blocks128(x, pow2):
    """1x128 blocks: e4m3 values and their scale (amax / 448, or the smallest power of two not below it)."""
    b = x.double().reshape(x.shape[0], -1, 128)
    s = (b.abs().amax(-1) / 448.0).float().double()
    if pow2:
        s = torch.exp2(torch.ceil(torch.log2(s)))
    s = torch.where(s > 0, s, torch.ones_like(s))
    q = (b / s[..., None]).float().clamp(-448.0, 448.0).to(torch.float8_e4m3fn).double()
    return q.reshape(x.shape), s


def _times_scale(q, s):
    return (q.reshape(*s.shape, 128) * s[..., None]).reshape(q.shape)


def _weight64(q, s):
    n, k = q.shape
    return (q.view(torch.float8_e4m3fn).double().reshape(n // 128, 128, k // 128, 128) * s.double()[:, None, :, None]).reshape(n, k)


def _grouped_choice64(x, gate_w, bias, K):
    s = torch.sigmoid(x @ gate_w.double().T)
    c = s + bias.double()
    E = c.shape[1]
    groups = c.reshape(-1, N_GROUP, E // N_GROUP)
    kept = groups.topk(min(2, E // N_GROUP), dim=2).values.sum(2).topk(TOPK_GROUP, dim=1).indices
    open_ = torch.zeros(groups.shape[:2], dtype=torch.bool, device=DEV).scatter_(1, kept, True)
    c = torch.where(open_.repeat_interleave(E // N_GROUP, dim=1), c, torch.full_like(c, -math.inf))
    ids = c.topk(K, dim=1).indices
    w = s.gather(1, ids)
    return ids, w / w.sum(1, keepdim=True) * ROUTED_SCALE


def _experts64(x, ids, w, weights, pow2=None):
    """sum over a row's experts of w * W2 quant(silu(W1g x) * W1u x); pow2 None: no quantisation in between."""
    out = torch.zeros_like(x)
    for e in range(len(weights)):
        row, slot = (ids == e).nonzero(as_tuple=True)
        if len(row) == 0:
            continue
        w1, w2 = weights[e]
        h = x[row] @ w1.T
        I = h.shape[1] // 2
        a = torch.nn.functional.silu(h[:, :I]) * h[:, I:]
        if pow2 is not None:
            a = _times_scale(*_blocks128(a, pow2))
        out.index_add_(0, row, (a @ w2.T) * w[row, slot][:, None])
    return out


class _Fp8Experts:
    def __init__(self, w1q, w1s, w2q, w2s):
        self.t = (w1q, w1s, w2q, w2s)

    def __len__(self):
        return self.t[0].shape[0]

    def __getitem__(self, e):
        w1q, w1s, w2q, w2s = self.t
        return _weight64(w1q[e], w1s[e]), _weight64(w2q[e], w2s[e])


def _attend64(q, k, v):
    p = torch.softmax((q @ k.T) / math.sqrt(q.shape[1]), dim=1)
    return p @ v


def exact(case, seed):
    c = case
    kind = c["kind"]
    if kind == "moe_f32":
        s = prepare(c, seed)
        x = s["x"].double()
        p, ids = torch.softmax(x @ s["wg"].double().T, dim=1).topk(c["K"], dim=1)
        return _experts64(x, ids, p / p.sum(1, keepdim=True), [(a.double(), b.double()) for a, b in zip(s["w1"], s["w2"])])
    if kind == "dsa_f32":
        s = prepare(c, seed)
        k, v = torch.cat([s["kc"], s["kp"]], 1).double(), s["v"].double()
        q = torch.cat([s["qn"], s["qp"]], 2).double()
        return torch.stack([_attend64(q[i], k[s["idx"][i].long()], v[s["idx"][i].long()]) for i in range(c["Q"])])
    if kind == "moe_fp8":
        gate_w, bias, *experts = _fp8_weights(c, seed)
        pow2 = c["option"] == "pow2"
        xq, xs = _blocks128(_normal((c["T"], c["D"]), seed * 16 + 5, 1.0), pow2)
        x = _times_scale(xq, xs)
        ids, w = _grouped_choice64(x, gate_w, bias, c["K"])
        return None, xs, _experts64(x, ids, w, _Fp8Experts(*experts), pow2)
    if kind == "experts":
        s = prepare(c, seed)
        _, _, *experts = _fp8_weights(c, seed)
        x = _times_scale(s["xq"].view(torch.float8_e4m3fn).double(), s["xs"].double())
        return _experts64(x, s["rid"], s["rw"].double(), _Fp8Experts(*experts), False)
    valid, table, pos, N = _decode_ids(c, seed)
    s = prepare(c, seed)
    kc, kp, v = (_normal((N, d), seed * 16 + i, 0.5, torch.bfloat16) for i, d in enumerate((512, 64, 512)))
    out = []
    for i in range(c["Q"]):
        p = pos[i][pos[i] >= 0]
        r = table[i][p // 64].long() * 64 + p % 64
        q = torch.cat([s["qn"][i], s["qp"][i]], 1).double()
        out.append(_attend64(q, torch.cat([kc[r], kp[r]], 1).double(), v[r].double()))
    return torch.stack(out)


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def work(case):
    c = case
    kind = c["kind"]
    if kind == "moe_f32":
        T, E, K, D, I = c["T"], c["E"], c["K"], c["D"], c["I"]
        return {"bytes": 4 * (2 * T * D + E * D + 3 * E * D * I), "flops": 2 * T * E * D + 6 * T * K * D * I}
    if kind == "dsa_f32":
        Q, H, Dc, Dp, S = c["Q"], c["H"], c["Dc"], c["Dp"], c["S"]
        return {"bytes": 4 * (Q * S * (2 * Dc + Dp + 1) + Q * H * (2 * Dc + Dp)), "flops": 2 * Q * H * S * (2 * Dc + Dp)}
    if kind in ("moe_fp8", "experts"):
        E, K, D, I = c["E"], c["K"], c["D"], c["I"]
        rows, per = (c["T"], K) if kind == "moe_fp8" else (c["R"], 2)
        active = E * (1.0 - (1.0 - per / E) ** rows)            # experts that at least one row reaches
        weights = active * (3 * D * I + 4 * 3 * (D // 128) * (I // 128))
        acts = rows * (D + D // 32) + 4 * rows * D
        b, f = weights + acts, 6.0 * rows * per * D * I
        if kind == "moe_fp8":
            b, f = b + 4 * rows * D + 4 * E * D, f + 2.0 * rows * E * D      # fp32 activations in, router weights
        else:
            b += 8 * rows * K
        return {"bytes": b, "flops": f}
    Q, H, S = c["Q"], c["H"], c["S"]
    mean = 0.5 * (c["seq_min"] + c["seq_max"])
    n = S if c["seq_min"] >= S else min(S, mean)
    return {"bytes": Q * n * 1088 * 2 + Q * H * 576 * 2 + Q * H * 512 * 4 + 4 * Q * S, "flops": 2.0 * Q * H * n * 1088}


def tolerance(case):
    """About four times the largest difference seen against the same sequence in 64-bit sums: fp32 layers 8e-7 to
    9e-7 (max 6e-6), bf16 decode 1.6e-3 (max 8e-3; the probabilities are rounded to bf16 before P*V), FP8 layer
    5e-5 to 8e-5 (max 3e-3; an activation near the middle of two e4m3 codes rounds either way)."""
    kind = case["kind"]
    if kind in ("moe_f32", "dsa_f32"):
        return {"rel": 4e-6, "max": 3e-5}
    if kind == "dsa_bf16":
        return {"rel": 6.5e-3, "max": 0.04}
    return {"rel": 3.5e-4, "max": 0.015}
