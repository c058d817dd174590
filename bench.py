"""Benchmark of the MSAQ-signed decode hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference] [--batch B]
    python -m torch.distributed.run --nnodes=1 --nproc-per-node N --master-addr 127.0.0.1 \\
        --master-port P bench.py --gpus N --steps K --warmup W

One step = one decode step of a Llama-3.1-70B-shaped decoder layer on packed
u4/gs2 weights, tensor-parallel over N GPUs: QKV GEMV -> K/V append (keys
Hadamard-rotated) -> GQA flash-decode over Lk cached keys -> O GEMV -> all-reduce
-> gate/up GEMV -> SiLU*mul -> down GEMV -> all-reduce.  Total work is fixed as N
grows (strong scaling).  The metric is achieved HBM bandwidth on ALGORITHMIC
bytes (packed codes + scales + activations of every op of the step, summed over
ranks) divided by the device-timed step, max over ranks.

Rank 0 prints ONE JSON line.  At N=1 the line also carries `detail`: per-op
microseconds and GB/s for the single-GPU configurations (Llama-3.1-8B GEMV
shapes at u in {2,3,4}, M in {1,4,16,64}; MHA and GQA flash-decode), a
`roofline` object for the dominant kernel and the CPU oracle timed beside it.
"""

import argparse
import json
import os
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

NOMINAL_PEAK_GBS = 8000.0
FALLBACK_PEAK_GBS = 6650.0
U, GS = 4, 2
LK = 8192                     # cached keys per sequence of the layer step
L2_BYTES = 126 << 20

# DRAM bytes (read + write) per launch of the dominant kernel from one ncu capture (`--case gemv` below) of
# `gemv_u4gs2_mma_kernel` on the 28672 x 4096 u4/gs2 M=1 GEMV: 91.85 MB read + 4.69 MB written (split-K partials).
# The kernel reads every packed byte once, so the figure scales with the algorithmic bytes; it has to be
# re-captured when the kernel's data flow changes.
NCU_TRAFFIC = {"kernel": "gemv_u4gs2_mma_kernel", "shape": [28672, 4096], "bytes_per_launch": 91.85e6 + 4.69e6,
               "algorithmic_bytes": 91.82e6}


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=None, help="default 200 (reference arm: 10)")
    ap.add_argument("--warmup", type=int, default=None, help="default 20 (reference arm: 2)")
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--batch", type=int, default=1)
    ap.add_argument("--no-detail", action="store_true")
    ap.add_argument("--case", default=None, choices=["gemv", "gemv16", "gemv128", "small", "pack", "kv", "layer"],
                    help="run a few launches of one op only (small driver for ncu captures)")
    a = ap.parse_args()
    if a.steps is None:
        a.steps = 200 if a.impl == "ours" else 10
    if a.warmup is None:
        a.warmup = 20 if a.impl == "ours" else 2
    return a


def measured_peak():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_PEAK_GBS, "fallback"


# --------------------------------------------------------------------------
# clocks
# --------------------------------------------------------------------------
class ClockSampler:
    """Samples SM clock and throttle reasons of one GPU through NVML while a region runs."""

    BITS = {0x8: "hw_slowdown", 0x40: "hw_thermal_slowdown", 0x20: "sw_thermal_slowdown", 0x4: "sw_power_cap"}

    def __init__(self, index):
        self.samples, self.reasons, self.max_mhz = [], set(), None
        self._stop = threading.Event()
        self._thread = None
        try:
            import pynvml
            pynvml.nvmlInit()
            self._nv = pynvml
            self._h = pynvml.nvmlDeviceGetHandleByIndex(index)
            self.max_mhz = int(pynvml.nvmlDeviceGetMaxClockInfo(self._h, pynvml.NVML_CLOCK_SM))
        except Exception:
            self._nv = None

    def _once(self):
        nv = self._nv
        self.samples.append(int(nv.nvmlDeviceGetClockInfo(self._h, nv.NVML_CLOCK_SM)))
        try:
            r = int(nv.nvmlDeviceGetCurrentClocksEventReasons(self._h))
        except Exception:
            r = int(nv.nvmlDeviceGetCurrentClocksThrottleReasons(self._h))
        for bit, name in self.BITS.items():
            if r & bit:
                self.reasons.add(name)

    def __enter__(self):
        if self._nv is not None:
            def loop():
                while not self._stop.is_set():
                    try:
                        self._once()
                    except Exception:
                        pass
                    self._stop.wait(0.005)
            self._thread = threading.Thread(target=loop, daemon=True)
            self._thread.start()
        return self

    def __exit__(self, *a):
        self._stop.set()
        if self._thread is not None:
            self._thread.join()

    def summary(self):
        s = sorted(self.samples)
        return {"sm_mhz": (s[len(s) // 2] if s else None), "sm_max_mhz": self.max_mhz,
                "reasons": sorted(self.reasons), "samples": len(s)}


# --------------------------------------------------------------------------
# building blocks
# --------------------------------------------------------------------------
def plane_bytes(u, gs):
    return 32 * (8 - u) // 8 + ((32 // gs) * u + 7) // 8 + 1


def gemv_bytes(OUT, K, M, u, gs):
    return OUT * (K // 32) * plane_bytes(u, gs) + 2 * K * M + 2 * OUT * M


def make_pack(OUT, K, u, gs, seed, dev):
    """Random bf16 ~N(0, 0.02) weight packed on the device -> pack dict holding the column-major planes."""
    import torch
    from ms_kernel_b200 import pack, tp
    g = torch.Generator(device=dev).manual_seed(seed)
    # pack in row chunks so that the bf16 source never needs more than ~1 GB
    rows = max(1, min(OUT, (512 << 20) // (2 * K)))
    parts = []
    for r0 in range(0, OUT, rows):
        W = (torch.randn((min(rows, OUT - r0), K), generator=g, device=dev) * 0.02).to(torch.bfloat16)
        p = pack.pack_weight(W, u, gs, device=dev)
        del p["upper"], p["shared"], W                 # the kernels read the column-major planes only
        parts.append(p)
    return parts[0] if len(parts) == 1 else tp.concat_rows(parts)


def make_linear(OUT, K, u, gs, seed, dev):
    from ms_kernel_b200 import ops
    return ops.PackedLinear(make_pack(OUT, K, u, gs, seed, dev), dev)


def graph_time(fns, iters, dev):
    """Capture `fns` (called in order) in one CUDA graph, replay `iters` times, return us per call of fns."""
    import torch
    s = torch.cuda.Stream(device=dev)
    s.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(s):
        for f in fns:
            f()
    torch.cuda.current_stream().wait_stream(s)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        for f in fns:
            f()
    for _ in range(3):
        g.replay()
    torch.cuda.synchronize()
    a, b = torch.cuda.Event(True), torch.cuda.Event(True)
    best = float("inf")
    for _ in range(3):
        a.record()
        for _ in range(iters):
            g.replay()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3 / iters / len(fns))
    return best


# --------------------------------------------------------------------------
# the layer step
# --------------------------------------------------------------------------
def layer_packs(shape, dev, seed):
    """One whole decoder layer, packed: the same bytes on every rank that uses the same seed."""
    d = shape.head_dim
    dims = {"q": (shape.n_q * d, shape.hidden), "k": (shape.n_kv * d, shape.hidden), "v": (shape.n_kv * d, shape.hidden),
            "o": (shape.hidden, shape.n_q * d), "gate": (shape.ffn, shape.hidden), "up": (shape.ffn, shape.hidden),
            "down": (shape.hidden, shape.ffn)}
    return {name: make_pack(OUT, K, U, GS, seed * 16 + i, dev) for i, (name, (OUT, K)) in enumerate(dims.items())}


def rope_tables_pos(pos, head_dim, dev):
    """cos, sin [1, head_dim/2] of one position, as the reference's harness builds them
    (tests/harness_batchsweep.py:124-129, theta = 500000)."""
    import torch
    inv = 1.0 / (500000.0 ** (torch.arange(0, head_dim, 2, device=dev).float() / head_dim))
    f = torch.outer(torch.tensor([float(pos)], device=dev), inv)
    return torch.cos(f).contiguous(), torch.sin(f).contiguous()


class LayerSet:
    """One rank's share of one decoder layer (weights + KV cache) and its graph.  The layer and the
    cache contents are generated whole from `seed` (identically on every rank) and then sharded, so
    that the tensor-parallel step can be compared with the single-GPU step on the same layer."""

    def __init__(self, shape, world, rank, B, dev, seed, all_reduce, packs=None, linears=None):
        import torch
        from ms_kernel_b200 import ops, tp
        self.B, self.shape, self.world, self.rank, self.seed, self.dev = B, shape, world, rank, seed, dev
        if linears is None:
            packs = packs if packs is not None else layer_packs(shape, dev, seed)
            local = tp.shard_layer(packs, shape, world, rank)
            linears = {name: ops.PackedLinear(p, dev) for name, p in local.items()}
        q, kv, f = shape.local(world)
        self.Lcap = LK + 16                    # capacity a multiple of 16: the tuned decode path
        self.cache = ops.KVCache(B, kv, shape.head_dim, self.Lcap, U, GS, dev, rotate=True)
        g = torch.Generator(device=dev).manual_seed(seed + 77)
        chunk = 2048
        for k0 in range(0, LK, chunk):
            # the whole batch x all kv heads, then this rank's heads: every rank draws the same numbers
            Kt = torch.randn((B, shape.n_kv, chunk, shape.head_dim), generator=g, device=dev).to(torch.bfloat16)
            Vt = torch.randn((B, shape.n_kv, chunk, shape.head_dim), generator=g, device=dev).to(torch.bfloat16)
            sl = slice(rank * kv, (rank + 1) * kv)
            self.cache.fill(Kt[:, sl].contiguous(), Vt[:, sl].contiguous(), key0=k0)
            del Kt, Vt
        self.layer = tp.DecoderLayerTP(shape, world, linears, self.cache, all_reduce)
        gh = torch.Generator(device=dev).manual_seed(seed + 99)
        self.h_in = torch.randn((B, shape.hidden), generator=gh, device=dev).to(torch.bfloat16)
        self.rope = rope_tables_pos(LK - 1, shape.head_dim, dev)
        self.h_out = None
        self.graph = None
        self.weight_bytes = sum(l.nbytes() for l in linears.values())
        torch.cuda.synchronize(dev)            # weights and cache complete before any step is enqueued (OPT_EARLY_WEIGHTS)

    def eager(self):
        # the step of the reference's decode_step (tests/harness_batchsweep.py:230-243): RoPE on q and k at the
        # new token's position, append to slot LK-1, attend LK keys
        return self.layer.step(self.h_in, LK - 1, LK, rope=self.rope)

    def capture(self):
        import torch
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            self.eager()
        torch.cuda.current_stream().wait_stream(s)
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.h_out = self.eager()

    def capture_e2e(self, h_host, out_host):
        """The same step with its host traffic inside the graph: pinned host -> device copy of the activations, the
        step, device -> pinned host copy of the result; one launch per step from the host."""
        import torch
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(s):
            self.h_in.copy_(h_host, non_blocking=True)
            out_host.copy_(self.eager(), non_blocking=True)
        torch.cuda.current_stream().wait_stream(s)
        torch.cuda.synchronize()
        self.graph_e2e = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph_e2e):
            self.h_in.copy_(h_host, non_blocking=True)
            out_host.copy_(self.eager(), non_blocking=True)


def timed_windows(replay, steps, barrier, reduce_max, min_total_ms=60.0, max_windows=40):
    """Device time of `steps` replays, as the best of several windows.

    A window: host barrier + device synchronise, one UNTIMED replay (its exchanges make every rank's
    stream wait for the slowest rank, so the timed region starts aligned on the device, whatever the
    host-side skew after the barrier), start event, exactly `steps` replays, stop event, synchronise.
    A window's time is the maximum over the ranks; windows repeat (at least three) until they add up to
    `min_total_ms`, so the result does not depend on how short `steps` makes one window."""
    import torch
    e0, e1 = torch.cuda.Event(True), torch.cuda.Event(True)
    times, total = [], 0.0
    while len(times) < 3 or (total < min_total_ms and len(times) < max_windows):
        barrier()
        replay(-1)
        e0.record()
        for i in range(steps):
            replay(i)
        e1.record()
        torch.cuda.synchronize()
        t = reduce_max(e0.elapsed_time(e1))
        times.append(t)
        total += t
    return min(times), times


def run_ours(args):
    import torch
    import torch.distributed as dist
    from ms_kernel_b200 import ops, tp

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world != args.gpus:
        raise SystemExit("--gpus %d but WORLD_SIZE=%d: launch with torch.distributed.run" % (args.gpus, world))
    ops._require()
    torch.cuda.set_device(local)
    dev = torch.device("cuda", local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", device_id=dev, timeout=datetime.timedelta(seconds=180))
    clocks = ClockSampler(local)               # NVML is opened here, well before any timed region

    def nccl_all_reduce(t):
        dist.all_reduce(t)
        return t

    shape = tp.LayerShape.llama31_70b()
    state = {"exchange": "none"}

    def make_all_reduce(B):
        if world == 1:
            return None
        mode = os.environ.get("MSAQ_BENCH_EXCHANGE", "push")
        if mode in ("push", "push_separate"):
            try:
                ar = tp.PeerExchange(dist.group.WORLD, B * shape.hidden, dev, fused=(mode == "push"))
                state["exchange"] = ("push over NVLink peer memory, plain peer stores of data words that carry the sequence "
                                     "number: " + ("issued by the O / down GEMVs' finishing warps tile by tile "
                                                   "(msaq_wonly_gemv_fused_push), then one wait-and-add kernel with the "
                                                   "residual add (msaq_peer_exchange)" if mode == "push" else
                                                   "one kernel after the GEMV (msaq_peer_exchange)"))
                return ar
            except Exception as e:
                state["exchange_note"] = "push exchange unavailable: %s" % str(e).splitlines()[0][:80]
                mode = "peer"
        if mode == "peer":
            try:
                ar = tp.peer_all_reduce(dist.group.WORLD, B * shape.hidden, torch.float32, dev)
                state["exchange"] = "one-shot all-reduce over NVLink peer memory (torch symmetric memory)"
                return ar
            except Exception as e:                              # keep NCCL, say why
                state["exchange"] = "nccl all-reduce (symmetric memory unavailable: %s)" % str(e).splitlines()[0][:80]
                return nccl_all_reduce
        state["exchange"] = "nccl all-reduce"
        return nccl_all_reduce

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    def reduce_max(x):
        if world == 1:
            return float(x)
        t = torch.tensor([float(x)], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    # the serving configuration: weights are packed once and complete before any step is enqueued, so the GEMVs may
    # fetch them ahead of the wait for the kernel in front (every LayerSet ends its construction with a synchronise)
    from ms_kernel_b200 import ops as _ops
    _ops.set_option(_ops.OPT_EARLY_WEIGHTS, True)
    B = args.batch
    all_reduce = make_all_reduce(B)
    packs0 = layer_packs(shape, dev, 1)
    probe = LayerSet(shape, world, rank, B, dev, 1, all_reduce, packs=packs0)
    per_rank_bytes = probe.layer.algorithmic_bytes(B, B * LK, U, GS)
    # rotate over enough distinct weight + cache sets that a step never finds its bytes in L2
    n_sets = max(1, -(-3 * L2_BYTES // max(1, per_rank_bytes)))
    n_sets = min(n_sets, 8)
    sets = [probe] + [LayerSet(shape, world, rank, B, dev, 2 + i, all_reduce) for i in range(n_sets - 1)]

    launches0 = torch.ops.msaq.launch_count()
    sets[0].eager()
    launches_per_step = int(torch.ops.msaq.launch_count() - launches0)
    for s in sets:
        s.capture()
    torch.cuda.synchronize()

    # ---- tensor-parallel parity: the sharded step against the single-GPU step on the same layer ----
    tp_parity = None
    if world > 1:
        for _ in range(4):                       # back-to-back replays: the exchange buffers rotate and are reused
            sets[0].graph.replay()
        torch.cuda.synchronize()
        if rank == 0:
            ref = LayerSet(shape, 1, 0, B, dev, 1, None, packs=packs0)
            h_ref = ref.eager().float()
            h_tp = sets[0].h_out.float()
            h0 = sets[0].h_in.float()
            tp_parity = float(((h_tp - h_ref).norm() / (h_ref - h0).norm()).item())
            finite = bool(torch.isfinite(h_tp).all().item())
            del ref, h_ref
            torch.cuda.empty_cache()
            if not finite or not tp_parity <= 2e-2:
                print(json.dumps({"error": "tensor-parallel step differs from the single-GPU step",
                                  "tp_parity_rel_fro": tp_parity, "finite": finite}), flush=True)
                os._exit(3)
        barrier()                                # nobody replays (and waits in an exchange) while rank 0 still checks
    del packs0

    for i in range(max(3, args.warmup)):
        sets[i % n_sets].graph.replay()

    def replay(i):
        sets[i % n_sets].graph.replay()

    with clocks:
        best_ms, windows = timed_windows(replay, args.steps, barrier, reduce_max)
    ms_per_step = best_ms / args.steps
    total_bytes = per_rank_bytes * world
    value = total_bytes / (ms_per_step * 1e-3) / 1e9

    # ---- end to end: the public API with host buffers in and out every step -------------------
    h_host = torch.randn((B, shape.hidden)).to(torch.bfloat16).pin_memory()
    out_host = torch.empty((B, shape.hidden), dtype=torch.bfloat16).pin_memory()

    for s in sets:
        s.capture_e2e(h_host, out_host)

    def e2e_step(i, eager):
        s = sets[i % n_sets]
        if eager:
            s.h_in.copy_(h_host, non_blocking=True)
            out_host.copy_(s.eager(), non_blocking=True)
        else:
            s.graph_e2e.replay()                  # copies and step captured from the same public calls: one launch per step
        torch.cuda.current_stream().synchronize()

    def e2e_time(eager, n):
        for i in range(3):
            e2e_step(i, eager)
        best = float("inf")
        for _ in range(3):
            barrier()
            t0 = time.perf_counter()
            for i in range(n):
                e2e_step(i, eager)
            best = min(best, reduce_max((time.perf_counter() - t0) * 1e3 / n))
        return best

    e2e_steps = max(args.steps, 200)
    e2e_ms_val = e2e_time(False, e2e_steps)
    e2e_eager_ms = e2e_time(True, e2e_steps)
    e2e_value = total_bytes / (e2e_ms_val * 1e-3) / 1e9

    peak, peak_kind = measured_peak()
    # ---- the dominant launch of the step, alone: this rank's gate+up GEMV (with its activation staging) ----
    gu = [st.layer.lin["gate_up"] for st in sets]
    gu_us = graph_time([(lambda l=l, st=st: l.fwd_fused(st.h_in, ops.PRO_RMSNORM)) for l, st in zip(gu, sets)], 20, dev)
    gu_bytes = gemv_bytes(gu[0].OUT, gu[0].K, B, U, GS)
    gu_gbs = gu_bytes / gu_us / 1e3
    roofline = {"bound": "hbm", "achieved": round(gu_gbs, 1), "peak": peak, "unit": "GB/s",
                "frac": round(gu_gbs / peak, 4), "peak_source": peak_kind + " copy bandwidth (burst)",
                "traffic": round(gu_bytes * NCU_TRAFFIC["bytes_per_launch"] / NCU_TRAFFIC["algorithmic_bytes"]),
                "traffic_source": "ncu dram bytes of the 28672x4096 launch, scaled by algorithmic bytes",
                "algorithmic_bytes": gu_bytes,
                "kernel": "gemv_u4gs2_mma_kernel with its activation staging: the layer's gate+up GEMV, %d x %d u4/gs2 M=%d"
                          % (gu[0].OUT, gu[0].K, B),
                "us_per_launch": round(gu_us, 2), "share_of_step": round(gu_us / (ms_per_step * 1e3), 3)}

    # ---- the same layer step at the other configured batch sizes (weights shared with the sets above) ----
    layer_detail = []
    for Bx in (8, 32):
        if Bx == B or args.no_detail:
            continue
        arx = make_all_reduce(Bx)
        bytes_x = tp.DecoderLayerTP(shape, world, sets[0].layer.lin, None, glue=sets[0].layer.glue).algorithmic_bytes(
            Bx, Bx * LK, U, GS)
        nx = int(max(1, min(n_sets, -(-3 * L2_BYTES // bytes_x))))
        xs = [LayerSet(shape, world, rank, Bx, dev, 1 + i, arx, linears=sets[i].layer.lin) for i in range(nx)]
        for x in xs:
            x.capture()
        for i in range(3):
            xs[i % nx].graph.replay()
        bx_ms, bx_windows = timed_windows(lambda i: xs[i % nx].graph.replay(), args.steps, barrier, reduce_max,
                                          min_total_ms=30.0)
        us = bx_ms / args.steps * 1e3
        layer_detail.append({"B": Bx, "Lk": LK, "us_per_step": round(us, 2),
                             "GBps": round(bytes_x * world / us / 1e3, 1),
                             "frac_of_%s_peak_per_gpu" % peak_kind: round(bytes_x / us / 1e3 / peak, 4),
                             "windows": len(bx_windows), "sets": nx})
        del xs
        torch.cuda.empty_cache()

    line = {
        "metric": "achieved_hbm_bandwidth_on_algorithmic_bytes", "value": round(value, 1), "unit": "GB/s",
        "n_gpus": world, "steps": args.steps, "warmup": max(3, args.warmup),
        "ms_per_step": round(ms_per_step, 5), "us_per_step": round(ms_per_step * 1e3, 2),
        "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
        "dtype": "u4 codes -> int8 MMA (M<=4, large M<=8) / exact bf16 MMA (above, tcgen05 for the largest batches), fp32 accumulate, bf16 in/out", "data": "synthetic",
        "config": {
            "workload": "llama-3.1-70b-shaped decoder layer, one decode step (RoPE on q and k included), u4/gs2 packed "
                        "weights and KV cache, hidden 8192, Hq 64, Hkv 8, D 128, FFN 28672, Lk %d, B %d" % (LK, B),
            "parallelism": "tp%d (rows of QKV/gate/up, K blocks of O/down, kv heads; 2 all-reduces per layer)" % world,
            "exchange": state["exchange"],
            "options": "MSAQ_OPT_EARLY_WEIGHTS=1 (weights packed at load, complete before the first step)",
            "l2": "rotating over %d distinct weight+cache sets (%.0f MB per GPU per set)" % (n_sets, per_rank_bytes / 1e6),
            "timing": "CUDA-graph replay per step; CUDA events on the launching stream around exactly `steps` replays, "
                      "barrier + synchronise on both sides, one untimed replay after the barrier to align the ranks on "
                      "the device; max over ranks per window, best of %d windows" % len(windows),
            "algorithmic_bytes_per_step": int(total_bytes),
        },
        "windows_ms": [round(w, 4) for w in windows],
        "tp_parity_rel_fro": tp_parity,
        "frac_of_nominal_8TBs_per_gpu": round(value / world / NOMINAL_PEAK_GBS, 4),
        "frac_of_%s_peak_per_gpu" % peak_kind: round(value / world / peak, 4),
        "clocks": clocks.summary(),
        "e2e": {"value": round(e2e_value, 1), "unit": "GB/s", "us_per_step": round(e2e_ms_val * 1e3, 1),
                "h2d_bytes_per_step": int(h_host.numel() * 2), "d2h_bytes_per_step": int(out_host.numel() * 2),
                "us_per_step_eager": round(e2e_eager_ms * 1e3, 1), "steps": e2e_steps,
                "api": "ms_kernel_b200.tp.DecoderLayerTP.step over ops.PackedLinear / ops.KVCache between a copy of the "
                       "activations from pinned host memory and a copy of the result to pinned host memory, all three "
                       "captured once in a CUDA graph and replayed per step (us_per_step_eager: the same calls launched "
                       "eagerly); wall clock with a stream sync per step, best of 3 runs"},
        "gpu_launches": launches_per_step * args.steps * len(windows),
        "gpu_launches_per_step": launches_per_step,
        "roofline": roofline,
    }
    if layer_detail:
        line["detail"] = {"layer": layer_detail}
    if world == 1 and rank == 0 and not args.no_detail:
        del sets, probe
        torch.cuda.empty_cache()
        extra = single_gpu_detail(dev, peak, peak_kind)
        line.setdefault("detail", {}).update(extra.pop("detail"))
        line.update(extra)
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        # Tearing the NCCL communicator down after CUDA-graph captured collectives can block for
        # minutes; every rank is past its last collective here, so leave without the teardown.
        dist.barrier()
        torch.cuda.synchronize()
        sys.stdout.flush()
        sys.stderr.flush()
        os._exit(0)


# --------------------------------------------------------------------------
# single-GPU detail: per-op numbers, roofline of the dominant kernel, CPU oracle
# --------------------------------------------------------------------------
def single_gpu_detail(dev, peak, peak_kind):
    import numpy as np
    import torch
    from ms_kernel_b200 import ops

    out = {"detail": {"gemv": [], "kv_decode": []}}
    shapes = [("qkv", 6144, 4096), ("o", 4096, 4096), ("gate_up", 28672, 4096), ("down", 4096, 14336)]
    for u in (4, 3, 2):
        for name, OUT, K in shapes:
            nbytes = OUT * (K // 32) * plane_bytes(u, GS)
            copies = max(2, -(-3 * L2_BYTES // nbytes))
            lins = [make_linear(OUT, K, u, GS, 31 * c + u, dev) for c in range(copies)]
            for M in (1, 4, 16, 64):
                x = torch.randn((M, K) if M > 1 else (K,), device=dev).to(torch.bfloat16)
                usec = graph_time([(lambda l=l: l.fwd(x)) for l in lins], 10, dev)
                b = gemv_bytes(OUT, K, M, u, GS)
                gbs = b / usec / 1e3
                out["detail"]["gemv"].append({"u": u, "gs": GS, "shape": name, "OUT": OUT, "K": K, "M": M,
                                              "us": round(usec, 2), "GBps": round(gbs, 1),
                                              "frac_8TBs": round(gbs / NOMINAL_PEAK_GBS, 3)})
            del lins
            torch.cuda.empty_cache()

    def kv_case(tag, B, Hq, Hkv, Lk, varlen):
        D = 128
        rng = np.random.default_rng(5)
        lens = rng.integers(Lk // 2, Lk + 1, size=B).astype(np.int32) if varlen else np.full(B, Lk, np.int32)
        per_key = 2 * Hkv * (D // 32) * plane_bytes(U, GS)
        nbytes = int(lens.sum()) * per_key
        copies = int(max(1, min(6, -(-3 * L2_BYTES // max(nbytes, 1)))))
        caches = []
        g = torch.Generator(device=dev).manual_seed(9)
        for _ in range(copies):
            c = ops.KVCache(B, Hkv, D, Lk + 16, U, GS, dev, rotate=True)
            step_keys = 4096 if B <= 16 else 1024
            for k0 in range(0, Lk, step_keys):
                n = min(step_keys, Lk - k0)
                Kt = torch.randn((B, Hkv, n, D), generator=g, device=dev)
                Kt[..., [3, 40, 77, 120]] *= 20
                c.fill(Kt.to(torch.bfloat16), torch.randn((B, Hkv, n, D), generator=g, device=dev).to(torch.bfloat16),
                       key0=k0)
                del Kt
            caches.append(c)
        q = torch.randn((B, Hq, D), generator=g, device=dev).to(torch.bfloat16)
        kn = torch.randn((B, Hkv, D), generator=g, device=dev).to(torch.bfloat16)
        sl = torch.from_numpy(lens).to(dev)
        pos = (sl - 1).to(torch.int32)

        def step(c):
            return c.append_attend(q, kn, kn, pos, Lk, sl)      # one new token per sequence, packed by the attention kernel

        usec = graph_time([(lambda c=c: step(c)) for c in caches], 10, dev)
        b = nbytes + 4 * B * Hq * D
        out["detail"]["kv_decode"].append({"case": tag, "B": B, "Hq": Hq, "Hkv": Hkv, "Lk": Lk, "varlen": varlen,
                                           "us": round(usec, 2), "GBps": round(b / usec / 1e3, 1),
                                           "frac_8TBs": round(b / usec / 1e3 / NOMINAL_PEAK_GBS, 3),
                                           "includes": "K/V append of one token (inside the attention kernel) + flash-decode"})
        del caches
        torch.cuda.empty_cache()

    for Hq in (8, 16):
        for Lk in (4096, 16384):
            kv_case("mha", 1, Hq, Hq, Lk, False)
    for Lk in (4096, 16384, 32768):
        for B in (1, 8, 16, 64):
            kv_case("gqa32/8", B, 32, 8, Lk, True)
    out["detail"]["msaq_over_mxint8"] = mxint8_ratio(dev, out["detail"])
    out["detail"]["reference_cuda"] = reference_cuda_anchor(dev, out["detail"])
    out["cpu_baseline"] = cpu_oracle_sample()
    return out


def mxint8_ratio(dev, detail):
    """The reference's headline metric (methodology.md:34-38): time of an MSAQ kernel over the time of its plain
    MXINT8 twin at the same optimisation level -- here the same pipelines with the sub-byte decode taken out.
    u4/gs2 moves 25 bytes per 32 values against MXINT8's 33, so 0.76 is what a purely bandwidth-bound pair gives."""
    import torch
    from ms_kernel_b200 import ops
    rows = []
    mine = {(r["OUT"], r["K"], r["M"]): r["us"] for r in detail["gemv"] if r["u"] == 4}
    for name, OUT, K in (("qkv", 6144, 4096), ("o", 4096, 4096), ("gate_up", 28672, 4096), ("down", 4096, 14336)):
        nbytes = OUT * (K // 32) * 33
        copies = max(2, -(-3 * L2_BYTES // nbytes))
        g = torch.Generator(device=dev).manual_seed(OUT + K)
        lins = []
        for c in range(copies):
            W = (torch.randn((OUT, K), generator=g, device=dev) * 0.02).to(torch.bfloat16)
            lins.append(ops.PackedLinearMX(W, dev))
            del W
        for M in (1, 4):
            x = torch.randn((M, K) if M > 1 else (K,), device=dev).to(torch.bfloat16)
            us = graph_time([(lambda l=l: l.fwd(x)) for l in lins], 10, dev)
            m = mine.get((OUT, K, M))
            rows.append({"op": "gemv", "shape": name, "OUT": OUT, "K": K, "M": M, "mxint8_us": round(us, 2), "msaq_us": m,
                         "msaq_over_mxint8": round(m / us, 3) if m else None})
        del lins
        torch.cuda.empty_cache()
    g = torch.Generator(device=dev).manual_seed(11)
    for B, Hq, Hkv, Lk in ((1, 8, 8, 16384), (1, 32, 8, 16384), (8, 32, 8, 16384), (16, 32, 8, 32768)):
        D = 128
        q = torch.randn((B, Hq, D), generator=g, device=dev).to(torch.bfloat16)
        res = {}
        for fmt in ("msaq", "mxint8"):
            per_key = 2 * Hkv * 4 * (25 if fmt == "msaq" else 33)
            copies = int(max(1, min(6, -(-3 * L2_BYTES // (B * Lk * per_key)))))
            caches = []
            for _ in range(copies):
                c = ops.KVCache(B, Hkv, D, Lk, U, GS, dev, rotate=False) if fmt == "msaq" else ops.KVCacheMX(B, Hkv, D, Lk, dev)
                for k0 in range(0, Lk, 4096):
                    n = min(4096, Lk - k0)
                    c.fill(torch.randn((B, Hkv, n, D), generator=g, device=dev).to(torch.bfloat16),
                           torch.randn((B, Hkv, n, D), generator=g, device=dev).to(torch.bfloat16), key0=k0)
                caches.append(c)
            res[fmt] = graph_time([(lambda c=c: c.attend(q, Lk)) for c in caches], 10, dev)
            del caches
            torch.cuda.empty_cache()
        rows.append({"op": "kv_decode", "B": B, "Hq": Hq, "Hkv": Hkv, "Lk": Lk, "mxint8_us": round(res["mxint8"], 2),
                     "msaq_us": round(res["msaq"], 2), "msaq_over_mxint8": round(res["msaq"] / res["mxint8"], 3)})
    return {"what": "u4/gs2 MSAQ kernel time over its plain-MXINT8 twin (same pipeline, no sub-byte decode); "
                    "bytes ratio 25/33 = 0.76; decode at full length, no append", "rows": rows}


def reference_cuda_anchor(dev, detail):
    """The reference project's own CUDA operators (its sm_86-era kernels rebuilt for sm_100a, oracle/_ref/) timed
    on this GPU by the same method, in a process of their own, beside this repository's numbers for the same
    shapes: a same-box anchor, not part of the product path.  Decode is timed at full length for both (the
    reference has one scalar Lk for the whole batch)."""
    import torch
    from ms_kernel_b200 import ops
    try:
        from oracle import ref_cuda
        if not ref_cuda.available():
            return {"unavailable": "oracle/_ref/ms_cuda_ref.so was not built (python oracle/build_ref.py needs the reference checkout)"}
        gemv_cases = [{"kind": "gemv", "OUT": OUT, "K": K, "M": M, "u": 4, "gs": 2}
                      for _, OUT, K in (("qkv", 6144, 4096), ("o", 4096, 4096), ("gate_up", 28672, 4096), ("down", 4096, 14336))
                      for M in (1, 4, 16, 64)]
        kv_cases = [{"kind": "kv_decode", "B": B, "Hq": Hq, "Hkv": Hkv, "Lk": Lk}
                    for B, Hq, Hkv, Lk in ((1, 8, 8, 4096), (1, 8, 8, 16384), (1, 16, 16, 16384), (1, 32, 8, 4096),
                                           (1, 32, 8, 16384), (8, 32, 8, 16384), (16, 32, 8, 32768))]
        torch.cuda.empty_cache()
        ref_us = ref_cuda.time_ops(gemv_cases + kv_cases)
    except Exception as e:                                      # the anchor must never take the benchmark down
        return {"unavailable": "reference CUDA run failed: %s" % str(e).splitlines()[-1][:200]}
    rows = []
    mine = {(r["OUT"], r["K"], r["M"]): r["us"] for r in detail["gemv"] if r["u"] == 4}
    for c, us in zip(gemv_cases, ref_us):
        m = mine.get((c["OUT"], c["K"], c["M"]))
        rows.append({"op": "wonly_gemv_wide" if c["M"] == 1 else "wonly_gemv_batched", "OUT": c["OUT"], "K": c["K"],
                     "M": c["M"], "reference_us": round(us, 2), "ours_us": m, "speedup": round(us / m, 2) if m else None})
    g = torch.Generator(device=dev).manual_seed(3)
    for c, us in zip(kv_cases, ref_us[len(gemv_cases):]):
        B, Hq, Hkv, Lk, D = c["B"], c["Hq"], c["Hkv"], c["Lk"], 128
        nbytes = B * Hkv * Lk * 2 * 4 * plane_bytes(U, GS)
        copies = int(max(1, min(6, -(-3 * L2_BYTES // nbytes))))
        caches = []
        for _ in range(copies):
            cch = ops.KVCache(B, Hkv, D, Lk, U, GS, dev, rotate=False)
            for k0 in range(0, Lk, 4096):
                n = min(4096, Lk - k0)
                cch.fill(torch.randn((B, Hkv, n, D), generator=g, device=dev).to(torch.bfloat16),
                         torch.randn((B, Hkv, n, D), generator=g, device=dev).to(torch.bfloat16), key0=k0)
            caches.append(cch)
        q = torch.randn((B, Hq, D), generator=g, device=dev).to(torch.bfloat16)
        m = graph_time([(lambda cc=cc: cc.attend(q, Lk)) for cc in caches], 10, dev)
        rows.append({"op": "kv_decode_attention_batched", "B": B, "Hq": Hq, "Hkv": Hkv, "Lk": Lk,
                     "reference_us": round(us, 2), "ours_us": round(m, 2), "speedup": round(us / m, 2)})
        del caches
        torch.cuda.empty_cache()
    return {"what": "the reference's own CUDA operators rebuilt for sm_100a (oracle/build_ref.py), same timing method, "
                    "own process; u4/gs2; decode at full length, no append", "rows": rows}


def cpu_oracle_sample():
    """The NumPy oracle on this box's host cores: W-only GEMV 4096x4096 u4/gs2 M=1."""
    import numpy as np
    import torch
    from ms_kernel_b200 import pack
    from oracle import msaq_oracle as orc

    OUT = K = 4096
    rng = np.random.default_rng(0)
    W = torch.from_numpy((rng.standard_normal((OUT, K)) * 0.02).astype(np.float32)).to(torch.bfloat16)
    p = pack.to_numpy(pack.pack_weight(W.cuda(), U, GS)) if torch.cuda.is_available() else orc.pack_weight(
        W.float().numpy(), U, GS)
    x = orc.to_bf16(rng.standard_normal((1, K)).astype(np.float32))
    orc.wonly_matmul(p, x)
    times = []
    t_end = time.perf_counter() + 15.0
    while len(times) < 3 or (time.perf_counter() < t_end and len(times) < 8):
        t0 = time.perf_counter()
        orc.wonly_matmul(p, x)
        times.append(time.perf_counter() - t0)
    best = min(times)
    Wdq = orc.dequant_weight(p)
    t0 = time.perf_counter()
    for _ in range(5):
        orc.wonly_matmul_predequant(Wdq, x)
    hoisted = (time.perf_counter() - t0) / 5
    b = gemv_bytes(OUT, K, 1, U, GS)
    return {"value": round(b / best / 1e9, 5), "unit": "GB/s", "cores": os.cpu_count(), "kind": "port",
            "sample": "oracle.wonly_matmul (dequantises the packed weight on every call, as the reference's NumPy "
                      "oracle does) on W-only GEMV 4096x4096 u4/gs2 M=1, best of %d calls" % len(times),
            "seconds_per_op": round(best, 4), "seconds_per_op_dequant_hoisted": round(hoisted, 5),
            "numpy": np.__version__}


# --------------------------------------------------------------------------
# reference arm: the CPU oracle on the host cores, same metric and config
# --------------------------------------------------------------------------
def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    import numpy as np
    from ms_kernel_b200 import tp
    from oracle import msaq_oracle as orc

    shape = tp.LayerShape.llama31_70b()
    B = args.batch
    # bounded sample of the step: a 1/32 slice of every GEMV's output rows and one kv head's decode over Lk/8 keys
    rng = np.random.default_rng(0)
    frac_rows, frac_keys = 32, 8
    mats = {name: (max(32, OUT // frac_rows), K) for name, (OUT, K) in shape.weight_shapes_local(1).items()}
    packs = {n: orc.pack_weight(orc.to_bf16((rng.standard_normal(s) * 0.02).astype(np.float32)), U, GS)
             for n, s in mats.items()}
    xs = {n: orc.to_bf16(rng.standard_normal((B, s[1])).astype(np.float32)) for n, s in mats.items()}
    Lk = LK // frac_keys
    Kc = orc.pack_kv(orc.to_bf16(rng.standard_normal((1, Lk, shape.head_dim)).astype(np.float32)), U, GS)
    Vc = orc.pack_kv(orc.to_bf16(rng.standard_normal((1, Lk, shape.head_dim)).astype(np.float32)), U, GS)
    qh = orc.to_bf16(rng.standard_normal((shape.n_q // shape.n_kv, shape.head_dim)).astype(np.float32))
    sample_bytes = sum(gemv_bytes(s[0], s[1], B, U, GS) for s in mats.values()) \
        + B * (Lk * 2 * 4 * plane_bytes(U, GS) + 4 * qh.size)

    def step():
        for n in mats:
            orc.wonly_matmul(packs[n], xs[n])
        kp = (Kc["scale_exp"], Kc["upper"], Kc["shared"])
        vp = (Vc["scale_exp"], Vc["upper"], Vc["shared"])
        for _ in range(B):
            orc.decode_attention_planes(qh, kp, vp, U, GS, Lk)

    for _ in range(args.warmup):
        step()
    steps = max(1, args.steps)
    t0 = time.perf_counter()
    for _ in range(steps):
        step()
    sec = (time.perf_counter() - t0) / steps
    value = sample_bytes / sec / 1e9
    sample = ("NumPy oracle port on the host cores: 1/%d of the output rows of each of the four layer GEMVs and one "
              "kv head's decode over Lk/%d keys per sequence; %d timed passes" % (frac_rows, frac_keys, steps))
    line = {
        "impl": "reference", "metric": "achieved_hbm_bandwidth_on_algorithmic_bytes", "value": round(value, 5),
        "unit": "GB/s", "n_gpus": args.gpus, "steps": steps, "warmup": args.warmup,
        "ms_per_step": round(sec * 1e3, 3), "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
        "dtype": "float64 (NumPy)", "data": "synthetic",
        "config": {"workload": "llama-3.1-70b-shaped decoder layer, one decode step, u4/gs2, Lk %d, B %d -- a BOUNDED "
                               "SAMPLE of it per step: 1/%d of the output rows of each of the four GEMVs and one kv head's "
                               "decode over Lk/%d keys per sequence (the NumPy oracle needs about a minute for the whole "
                               "step); GB/s on the sample's own algorithmic bytes" % (LK, B, frac_rows, frac_keys)},
        "cpu_baseline": {"value": round(value, 5), "unit": "GB/s", "cores": os.cpu_count(), "kind": "port",
                         "sample": sample},
        "e2e": {"value": round(value, 5), "unit": "GB/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)


def run_case(args):
    """A handful of launches of one op on cuda:0: the 28672x4096 u4/gs2 GEMV with one, 16 or 128 rows (92 MB per launch), the
    GEMVs of one wave (4096x14336 with one row and with eight, 46 MB), loading (packing 14336x4096, a prompt of 8 x 8191 keys, widening
    4096x14336 to bf16), the GQA 32/8 flash-decode at Lk=16384, B=8 (157 MB) or the layer step.  Meant to be run under ncu."""
    import torch
    from ms_kernel_b200 import ops
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(0)
    g = torch.Generator(device=dev).manual_seed(1)
    if args.case == "layer":
        # three eager decode steps of the 70B-shaped layer on one GPU (the launch list of a step)
        from ms_kernel_b200 import tp
        shape = tp.LayerShape.llama31_70b()
        ops.set_option(ops.OPT_EARLY_WEIGHTS, True)         # as the timed bench runs
        sets = [LayerSet(shape, 1, 0, args.batch, dev, 1 + i, None) for i in range(2)]
        torch.cuda.synchronize()
        for i in range(3):
            y = sets[i % 2].eager()
    elif args.case == "small":
        lins = [make_linear(4096, 14336, U, GS, 3 + i, dev) for i in range(4)]
        x = torch.randn((8, 14336), generator=g, device=dev).to(torch.bfloat16)
        for i in range(12):                                 # integer and bf16 direct kernels in turn
            y = lins[i % 4].fwd(x[0] if i & 1 else x)
    elif args.case == "pack":
        from ms_kernel_b200 import pack
        W = (torch.randn((14336, 4096), generator=g, device=dev) * 0.02).to(torch.bfloat16)
        K, V = (torch.randn((1, 8, 8191, 128), generator=g, device=dev).to(torch.bfloat16) for _ in range(2))
        cache = ops.KVCache(1, 8, 128, 8192, U, GS, dev, rotate=True)
        lins = [make_linear(4096, 14336, U, GS, 3 + i, dev) for i in range(3)]
        for lin in lins:
            p = pack.pack_weight(W, U, GS, device=dev)
            cache.fill(K, V)
            y = torch.ops.msaq.ms_dequant_bf16(lin.scale_exp, lin.upper_cm, lin.shared_cm, lin.OUT, lin.K, lin.nb, lin.u, lin.gs)
    elif args.case in ("gemv", "gemv16", "gemv128"):
        lins = [make_linear(28672, 4096, U, GS, 3 + i, dev) for i in range(4)]
        M = {"gemv": 1, "gemv16": 16, "gemv128": 128}[args.case]      # integer MMA, register operands, tcgen05 / tensor memory
        x = torch.randn((M, 4096) if M > 1 else (4096,), generator=g, device=dev).to(torch.bfloat16)
        for i in range(6):
            y = lins[i % 4].fwd(x)
    else:
        B, Hq, Hkv, Lk, D = 8, 32, 8, 16384, 128
        caches = []
        for _ in range(2):
            c = ops.KVCache(B, Hkv, D, Lk, U, GS, dev, rotate=True)
            for k0 in range(0, Lk, 4096):
                c.fill(torch.randn((B, Hkv, 4096, D), generator=g, device=dev).to(torch.bfloat16),
                       torch.randn((B, Hkv, 4096, D), generator=g, device=dev).to(torch.bfloat16), key0=k0)
            caches.append(c)
        q = torch.randn((B, Hq, D), generator=g, device=dev).to(torch.bfloat16)
        for i in range(6):
            y = caches[i % 2].attend(q, Lk)
    torch.cuda.synchronize()
    print(json.dumps({"case": args.case, "checksum": float(y.float().abs().sum())}))


if __name__ == "__main__":
    a = parse()
    if a.case:
        run_case(a)
    elif a.impl == "reference":
        run_reference(a)
    else:
        run_ours(a)
