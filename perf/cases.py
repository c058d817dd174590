"""Performance cases of the packed decode path: the calls a program that serves a model on packed weights and a packed
KV cache makes, through the package's public entry points, from the smallest to the largest.

A case is a dict of plain values; `kind` picks the call:

  linear   ops.PackedLinear.fwd on x [K] or [M, K] (weight-only GEMV and small-batch product)
  fill     ops.KVCache.fill (prefill: K rotated, K and V quantised into the cache)
  attend   ops.KVCache.append_attend (one decode step of attention: append the new token, attend the cache)
  layer    tp.DecoderLayerTP.step (one whole decoder-layer decode step on one GPU)
  pack     pack.pack_weight (loading: a bf16 weight to packed planes)
  dequant  torch.ops.msaq.ms_dequant_bf16 (prefill: a packed weight to the dense operand of a GEMM)

Inputs are synthetic: weights ~ N(0, 0.02) in bf16, activations, keys and values ~ N(0, 1) in bf16, a few key channels
larger than the rest.  `exact` computes the same results in 64 bits with plain torch: its own quantiser, its own
Hadamard rotation and RoPE, nothing of this package.
"""

import math

import torch

from ms_kernel_b200 import ops, pack, tp

DEV = "cuda"
GS = 2                      # the group size of every configuration of this repository
HEAD_DIM = 128
EPS = 1e-5


# ---------------------------------------------------------------------------------------------- the cases
def listed():
    return [
        # O projection of a Llama-3.1-8B-shaped layer, one token: the smallest GEMV, launch latency counts
        {"name": "linear 4096x4096 u4 M1", "kind": "linear", "OUT": 4096, "K": 4096, "u": 4, "M": 1},
        # gate+up of a Llama-3.1-70B-shaped layer, one token: the largest GEMV, streams 367 MB
        {"name": "linear 57344x8192 u4 M1", "kind": "linear", "OUT": 57344, "K": 8192, "u": 4, "M": 1},
        # gate+up of the 8B shape in the 5+3 bit format
        {"name": "linear 28672x4096 u3 M1", "kind": "linear", "OUT": 28672, "K": 4096, "u": 3, "M": 1},
        # down projection of the 8B shape in the 6+2 bit format, an odd handful of sequences
        {"name": "linear 4096x14336 u2 M5", "kind": "linear", "OUT": 4096, "K": 14336, "u": 2, "M": 5},
        # a batch of sixteen sequences through gate+up
        {"name": "linear 28672x4096 u4 M16", "kind": "linear", "OUT": 28672, "K": 4096, "u": 4, "M": 16},
        # continuous batching: a ragged batch through the fused QKV projection
        {"name": "linear 6144x4096 u4 M61", "kind": "linear", "OUT": 6144, "K": 4096, "u": 4, "M": 61},
        # prefill of one prompt of odd length into a GQA cache
        {"name": "fill 8x8191", "kind": "fill", "B": 1, "Hkv": 8, "L": 8191},
        # one long conversation: attention of one sequence, latency counts
        {"name": "attend 32/8 B1 16381", "kind": "attend", "B": 1, "Hq": 32, "Hkv": 8, "Lk": 16381},
        # many long conversations of different lengths: the largest attention call
        {"name": "attend 32/8 B16 32768", "kind": "attend", "B": 16, "Hq": 32, "Hkv": 8, "Lk": 32768},
        # a whole 8B-shaped layer, one token: five dependent calls, launches and host work count
        {"name": "layer 8b B1 4096", "kind": "layer", "B": 1, "Lk": 4096},
        # loading: quantise and pack one matrix
        {"name": "pack 14336x4096 u4", "kind": "pack", "OUT": 14336, "K": 4096, "u": 4},
        # prefill: the down projection widened once for the dense GEMMs of a long prompt
        {"name": "dequant 4096x14336 u4", "kind": "dequant", "OUT": 4096, "K": 14336, "u": 4},
    ]


def _log_int(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], its logarithm spread evenly."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi))) // step * step))) // step * step


def draw(rng):
    """Projections of 256 to 57344 rows (whole 16-row groups, as heads and FFN shards give) and 256 to 28672 columns
    (whole 32-blocks), any u, batches of 1 to 128; caches of any length, MHA and GQA, any ragged batch."""
    kind = rng.choice(["linear"] * 6 + ["fill", "attend", "attend", "layer", "pack", "dequant"])
    if kind == "linear":
        OUT = _log_int(rng, 256, 57344, 16)
        K = _log_int(rng, 256, min(28672, (57344 * 8192) // OUT), 32)
        M = rng.choice([1, 1, _log_int(rng, 2, 8), _log_int(rng, 9, 128)])
        return {"kind": kind, "OUT": OUT, "K": K, "u": rng.choice([4, 4, 3, 2]), "M": M}
    if kind == "fill":
        B, Hkv = rng.randint(1, 4), rng.choice([1, 2, 4, 8, 16])
        return {"kind": kind, "B": B, "Hkv": Hkv, "L": _log_int(rng, 17, 16384 * 8 // max(8, B * Hkv))}
    if kind == "attend":
        Hkv = rng.choice([1, 2, 4, 8, 16])
        Hq = Hkv * rng.choice([1, 2, 4, 8])
        B = _log_int(rng, 1, 16)
        return {"kind": kind, "B": B, "Hq": Hq, "Hkv": Hkv, "Lk": _log_int(rng, 100, min(32768, 8 * 16 * 32768 // (B * Hkv)))}
    if kind == "layer":
        return {"kind": kind, "B": rng.randint(1, 16), "Lk": _log_int(rng, 100, 8192)}
    OUT = _log_int(rng, 256, 28672, 16)
    K = _log_int(rng, 256, min(16384, 14336 * 4096 // OUT), 32)
    return {"kind": kind, "OUT": OUT, "K": K, "u": rng.choice([4, 4, 3, 2])}


# ---------------------------------------------------------------------------------------------- inputs
def _gen(seed, stream):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 64 + stream)


def _randn(shape, gen, scale=1.0):
    """bf16 values of N(0, scale)."""
    t = torch.randn(shape, generator=gen, device=DEV, dtype=torch.bfloat16)
    return t.mul_(scale) if scale != 1.0 else t


def _weight(OUT, K, seed, stream):
    return _randn((OUT, K), _gen(seed, stream), 0.02)


def _linear(OUT, K, u, seed, stream):
    p = pack.pack_weight(_weight(OUT, K, seed, stream), u, GS, device=DEV)
    del p["upper"], p["shared"]                          # the kernels read the column-major planes only
    return ops.PackedLinear(p, DEV)


def _keys_values(B, Hkv, L, seed):
    g = _gen(seed, 1)
    K, V = _randn((B, Hkv, L, HEAD_DIM), g), _randn((B, Hkv, L, HEAD_DIM), g)
    K[..., 5] *= 4                                       # keys have a few channels that are larger than the rest
    K[..., 77] *= 3
    return K, V


def _lens(case, seed):
    """Ragged lengths of a batch (the longest is Lk); one sequence attends all of its keys."""
    B, Lk = case["B"], case["Lk"]
    f = torch.rand(B, generator=torch.Generator().manual_seed(int(seed) * 64 + 7))
    lens = (Lk * (0.5 + 0.5 * f)).to(torch.int32).clamp(1, Lk)
    lens[0] = Lk
    return lens


def _rope_tables(rows, device=DEV):
    inv = 1.0 / (500000.0 ** (torch.arange(0, HEAD_DIM, 2, device=device).float() / HEAD_DIM))
    f = torch.outer(torch.arange(rows, device=device).float(), inv)
    return torch.cos(f).contiguous(), torch.sin(f).contiguous()


def _capacity(Lk):
    return (Lk + 15) // 16 * 16


def _attend_inputs(case, seed):
    B, Hq, Hkv = case["B"], case["Hq"], case["Hkv"]
    g = _gen(seed, 2)
    return (_randn((B, Hq, HEAD_DIM), g), _randn((B, Hkv, HEAD_DIM), g), _randn((B, Hkv, HEAD_DIM), g))


LAYER = (("qkv", 6144, 4096), ("o", 4096, 4096), ("gate_up", 28672, 4096), ("down", 4096, 14336))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        M, K = case["M"], case["K"]
        x = _randn((K,) if M == 1 else (M, K), _gen(seed, 1))
        return {"kind": kind, "lin": _linear(case["OUT"], K, case["u"], seed, 0), "x": x}
    if kind == "fill":
        K, V = _keys_values(case["B"], case["Hkv"], case["L"], seed)
        cache = ops.KVCache(case["B"], case["Hkv"], HEAD_DIM, _capacity(case["L"]), 4, GS, DEV)
        return {"kind": kind, "cache": cache, "K": K, "V": V}
    if kind == "attend":
        Lk = case["Lk"]
        cache = ops.KVCache(case["B"], case["Hkv"], HEAD_DIM, _capacity(Lk), 4, GS, DEV)
        K, V = _keys_values(case["B"], case["Hkv"], Lk, seed)
        cache.fill(K, V)
        q, k, v = _attend_inputs(case, seed)
        lens = _lens(case, seed).to(DEV)
        return {"kind": kind, "cache": cache, "q": q, "k": k, "v": v, "Lk": Lk, "lens": lens,
                "pos": (lens - 1).contiguous(), "rope": _rope_tables(_capacity(Lk))}
    if kind == "layer":
        B, Lk = case["B"], case["Lk"]
        shape = tp.LayerShape.llama31_8b()
        linears = {n: _linear(OUT, K, 4, seed, 8 + i) for i, (n, OUT, K) in enumerate(LAYER)}
        cache = ops.KVCache(B, shape.n_kv, HEAD_DIM, _capacity(Lk), 4, GS, DEV)
        cache.fill(*_keys_values(B, shape.n_kv, Lk, seed))
        lens = _lens(case, seed).to(DEV)
        return {"kind": kind, "layer": tp.DecoderLayerTP(shape, 1, linears, cache), "cache": cache,
                "h": _randn((B, shape.hidden), _gen(seed, 2)), "Lk": Lk, "lens": lens, "pos": (lens - 1).contiguous(),
                "rope": _rope_tables(_capacity(Lk))}
    if kind == "pack":
        return {"kind": kind, "W": _weight(case["OUT"], case["K"], seed, 0), "u": case["u"]}
    return {"kind": kind, "lin": _linear(case["OUT"], case["K"], case["u"], seed, 0)}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return state["lin"].fwd(state["x"])
    if kind == "fill":
        state["cache"].fill(state["K"], state["V"])
        return [*state["cache"].k, *state["cache"].v]
    if kind == "attend":
        c = state["cache"]
        out = c.append_attend(state["q"], state["k"], state["v"], state["pos"], state["Lk"], state["lens"], state["rope"])
        return [out, *c.k, *c.v]
    if kind == "layer":
        c = state["cache"]
        out = state["layer"].step(state["h"], state["pos"], state["Lk"], state["lens"], state["rope"])
        return [out, *c.k, *c.v]
    if kind == "pack":
        p = pack.pack_weight(state["W"], state["u"], GS, device=DEV)
        return [p["scale_exp"], p["upper"], p["shared"], p["upper_cm"], p["shared_cm"]]
    lin = state["lin"]
    return torch.ops.msaq.ms_dequant_bf16(lin.scale_exp, lin.upper_cm, lin.shared_cm, lin.OUT, lin.K, lin.nb, lin.u, lin.gs)


# ---------------------------------------------------------------------------------------------- what a pass needs
def _block_bytes(u):
    return 32 * (8 - u) // 8 + (32 // GS * u + 7) // 8 + 1


def _linear_work(OUT, K, M, u):
    return OUT * (K // 32) * _block_bytes(u) + 2 * M * (K + OUT), 2 * M * OUT * K


def _attend_work(B, Hq, Hkv, keys):
    """`keys`: attended keys, summed over the batch."""
    row = 2 * HEAD_DIM // 32 * _block_bytes(4)                                       # one key and one value row
    return keys * Hkv * row + B * (4 * Hq + 4 * Hkv) * HEAD_DIM + B * Hkv * row, 4 * keys * Hq * HEAD_DIM


def work(case):
    kind = case["kind"]
    if kind == "linear":
        b, f = _linear_work(case["OUT"], case["K"], case["M"], case["u"])
    elif kind == "fill":
        rows = 2 * case["B"] * case["Hkv"] * case["L"]
        b, f = rows * (2 * HEAD_DIM + HEAD_DIM // 32 * _block_bytes(4)), rows * HEAD_DIM * 8
    elif kind == "attend":
        b, f = _attend_work(case["B"], case["Hq"], case["Hkv"], 0.75 * case["B"] * case["Lk"] + 0.25 * case["Lk"])
    elif kind == "layer":
        b, f = _attend_work(case["B"], 32, 8, 0.75 * case["B"] * case["Lk"] + 0.25 * case["Lk"])
        for _, OUT, K in LAYER:
            wb, wf = _linear_work(OUT, K, case["B"], 4)
            b, f = b + wb, f + wf
    elif kind == "pack":
        n = case["OUT"] * case["K"]
        b, f = n * 2 + n // 32 * (2 * _block_bytes(case["u"]) - 1), n * 8            # both plane orders, one scale plane
    else:
        n = case["OUT"] * case["K"]
        b, f = n // 32 * _block_bytes(case["u"]) + n * 2, n * 2
    return {"bytes": float(b), "flops": float(f)}


def tolerance(case):
    kind = case["kind"]
    if kind in ("fill", "pack", "dequant"):
        return "exact"                                  # bytes, and products that are exact in bf16
    if kind == "layer":
        # bf16 between the steps; the new token's codes follow from a bf16 projection and may move by a rounding
        return {"rel": 1e-2, "max": 0.1, "differ": 1e-3}
    # one rounding of the result to bf16 (2^-9 of the value at most), the sums in 32 bits; the cache bytes are the same
    return {"rel": 6e-3, "max": 0.05}


# ---------------------------------------------------------------------------------------------- 64-bit results
def _quantise64(x, u):
    """The value of x [..., K] after the quantiser: per 32-block 2^(floor(log2 max|x|) - 6) as the grid, upper codes on
    2^u times the grid, one shared code for the mean residual of each pair."""
    b = x.double().reshape(*x.shape[:-1], -1, 32)
    amax = b.abs().amax(-1, keepdim=True).clamp_min(1e-30)
    e = (torch.frexp(amax).exponent - 1 - 6).clamp(-127, 127).double()
    fine = torch.exp2(e)
    coarse = fine * (1 << u)
    lim = (1 << (7 - u)) - 1
    up = torch.round(b / coarse).clamp(-lim, lim)
    res = (b - up * coarse).reshape(*b.shape[:-1], 32 // GS, GS)
    sh = torch.round(res.sum(-1) / GS / fine).clamp(-(1 << (u - 1)), (1 << (u - 1)) - 1)
    q = up * (1 << u) + sh.repeat_interleave(GS, -1)
    return (q * fine).reshape(x.shape)


def _hadamard(x):
    """The orthonormal Hadamard rotation of the last axis in fp32, stage by stage, as keys are rotated when written."""
    n = x.shape[-1]
    y = x.float()
    h = 1
    while h < n:
        z = y.reshape(*x.shape[:-1], n // (2 * h), 2, h)
        y = torch.stack((z[..., 0, :] + z[..., 1, :], z[..., 0, :] - z[..., 1, :]), -2).reshape(x.shape)
        h *= 2
    return y * torch.tensor(1.0 / math.sqrt(n), dtype=torch.float32, device=x.device)


def _rope(x, cos, sin):
    """x [B, heads, D]; cos, sin [B, D/2] in fp32: pairs (2j, 2j+1) rotated, rounded to bf16."""
    a, b = x.float()[..., 0::2], x.float()[..., 1::2]
    c, s = cos[:, None], sin[:, None]
    return torch.stack((a * c - b * s, a * s + b * c), -1).reshape(x.shape).to(torch.bfloat16)


def _matmul64(x, OUT, K, u, seed, stream):
    """x [M, K] times the quantised weight's transpose, in row chunks."""
    W = _weight(OUT, K, seed, stream)
    step = max(1, (1 << 26) // K)
    return torch.cat([x.double() @ _quantise64(W[r:r + step], u).T for r in range(0, OUT, step)], -1)


def _attention64(case, seed, Hq, Hkv, q, k, v):
    """Attention over the quantised cache with the new token in its slot, one sequence at a time."""
    B, Lk = case["B"], case["Lk"]
    lens = _lens(case, seed).tolist()
    cos, sin = _rope_tables(_capacity(Lk))
    at = torch.tensor([n - 1 for n in lens], device=DEV)
    q, k = _rope(q, cos[at], sin[at]), _rope(k, cos[at], sin[at])
    K, V = _keys_values(B, Hkv, Lk, seed)
    out = torch.empty((B, Hq, HEAD_DIM), dtype=torch.float64, device=DEV)
    for b in range(B):
        K[b, :, lens[b] - 1], V[b, :, lens[b] - 1] = 0, 0
        for h in range(Hkv):
            Kh, Vh = K[b, h, : lens[b]].float(), V[b, h, : lens[b]]
            Kh = _hadamard(Kh)
            Kh[-1] = _hadamard(k[b, h].float())
            Vh[-1] = v[b, h]
            Kq, Vq = _quantise64(Kh, 4), _quantise64(Vh, 4)
            G = Hq // Hkv
            s = _hadamard(q[b, h * G:(h + 1) * G]).double() @ Kq.T / math.sqrt(HEAD_DIM)
            out[b, h * G:(h + 1) * G] = torch.softmax(s, -1) @ Vq
    return out


def _rmsnorm64(x):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + EPS)


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        M, K = case["M"], case["K"]
        x = _randn((K,) if M == 1 else (M, K), _gen(seed, 1))
        y = _matmul64(x.reshape(M, K), case["OUT"], K, case["u"], seed, 0)
        return y.reshape(-1) if M == 1 else y
    if kind == "dequant":
        return _quantise64(_weight(case["OUT"], case["K"], seed, 0), case["u"]).T.contiguous()
    if kind == "attend":
        return [_attention64(case, seed, case["Hq"], case["Hkv"], *_attend_inputs(case, seed))] + [None] * 6
    if kind == "layer":
        B = case["B"]
        h = _randn((B, 4096), _gen(seed, 2)).double()
        mm = lambda x, i: _matmul64(x, LAYER[i][1], LAYER[i][2], 4, seed, 8 + i)  # noqa: E731
        qkv = mm(_rmsnorm64(h), 0)
        q, k, v = (t.reshape(B, -1, HEAD_DIM) for t in qkv.split([4096, 1024, 1024], -1))
        a = _attention64(case, seed, 32, 8, q, k, v.to(torch.bfloat16))
        h = h + mm(a.reshape(B, -1), 1)
        gate, up = mm(_rmsnorm64(h), 2).chunk(2, -1)
        return [h + mm(torch.nn.functional.silu(gate) * up, 3)] + [None] * 6
    return None
