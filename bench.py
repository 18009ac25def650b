"""Benchmark of the ciphertext-arithmetic hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl b200|reference] [--streams S]

Workload (the batched CKKS evaluation the headline metric is quoted on):
CKKS, N = 16384, coefficient modulus chain {60, 40 x 7, 60} bits (8 data limbs and
one special prime), 64 ciphertext pairs per step. Each pair goes through
multiply -> relinearize -> rescale_to_next -> rotate_vector(k) over 13 Galois keys,
k in {1, 2, 4, ..., 4096}, each step taken by as many pairs as pairs i with
i mod 13 == log2 k (the pairs of a step consecutive inside each sub-batch, so one
grouped Galois call serves all 13 keys; seal-cuda_b200/python/ckks_step.py, the
same step the GPU parity test checks word for word). One op = one pair through
that chain. Inputs and keys are seeded, uniformly random residues modulo each
prime (the arithmetic performed is the same as on encrypted data).

* ``value``: ops/s with inputs resident in HBM (CUDA events on the launch stream,
  max over ranks). Inputs (2 x 128 MB) exceed the 126 MB L2 between steps. Each
  step's 64 pairs run as S concurrent sub-batches, one stream each (default 2), the
  whole fork/join captured once as a CUDA graph and replayed per step (--no-graph:
  eager launches).
* ``e2e``: the same metric through the C ABI with host buffers: every step copies
  both operand batches from pinned host memory and reads the results back, as 2
  sub-batches whose copies run on one stream per direction, overlapping the
  neighbouring sub-batches' arithmetic (three device buffer sets, ordered by events).
* ``roofline``: the dominant kernel from the library's per-launch event trace of the
  same steps run as one batch on one stream, against the measured HBM copy peak and
  (``roofline.arith``) the measured arithmetic ceiling of the transforms.
* ``cpu_baseline``: the reference's own CPU implementation (compiled under
  oracle/_ref) on a bounded sample of the same workload, one process per core.
* ``plain_per_op``: the same chain driven one pair per call (batch 1), as the
  reference's evaluator is used; ``batched_over_per_op`` is the batching gain.
* ``reference_gpu_per_op``: the reference's own CUDA evaluator (its sources compiled
  for sm_100a under oracle/_ref by oracle/Makefile) on the same workload, one pair
  per call, in a child process; ``batched_over_reference_gpu_per_op`` compares.
* ``ntt_sweep``: the raw NTT / dyadic / inverse NTT workload (256 x 8 limbs, N =
  4096 .. 32768) with GB/s and fraction of the measured copy peak per kernel, and of
  the FP64 ceiling per transform.
* ``uneven_batch``: 512 BFV/BGV ciphertexts of degrees 4096 / 8192 / 16384 through
  multiply, relinearize and rotate_rows as one captured CUDA graph, beside the
  one-ciphertext-per-call path.
* ``serving``: the serving loop (MatmulServer, BFV N = 8192, 5 primes): Poisson
  arrivals of encrypted vector x matrix requests at several rates plus a burst,
  p50/p99 latency and throughput per rate.

``--impl reference`` times only that CPU implementation as the benchmark line.
With ``--gpus N`` (torchrun, one rank per GPU) every rank runs an independent
replica of the workload; nothing is exchanged (weak scaling).
"""
from __future__ import annotations

import argparse
import ctypes
import json
import math
import multiprocessing as mp
import os
import statistics
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path[:0] = [os.path.join(ROOT, "seal-cuda_b200", "python"), os.path.join(ROOT, "oracle")]

N = 16384
BITS = [60] + [40] * 7 + [60]
DEFAULT_PAIRS = 64
PAIRS = DEFAULT_PAIRS
SCALE_BITS = 40
STEPS_K = [1 << i for i in range(13)]
METRIC = "HE mul+relin+rescale+rotate ops/s (CKKS N=16384, batched 64 pairs)"
WORKLOAD = "ckks_n16384_L8_batch64_mul_relin_rescale_rotate"
FALLBACK_HBM_GBS = 6650.0
PER_OP_PAIRS = 16
E2E_CHUNKS = 2   # sub-batches per step in the end-to-end copy pipeline
HEADLINE_SUB_BATCHES = 2   # concurrent sub-batches (one stream each) per step of `value`
# serving workload: encrypted vector x plaintext matrix (MatmulHelper coefficient
# encoding), BFV N = 8192, 5 primes, 20-bit batching t, Poisson arrivals
SERVE_N = 8192
SERVE_BITS = [43, 43, 44, 44, 44]
SERVE_RATES = [10, 200, 1000, 2000]


def _peak_hbm():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(p) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


# ------------------------------------------------------------ clocks sampler
class ClockSampler:
    """Samples the SM clock and the clock-event (throttle) reasons of the benchmark's
    GPU every 2 ms through NVML. start() returns once sampling runs; only the samples
    taken between mark() (the timed region's start) and stop() are reported, so even a
    region of a few tens of milliseconds gets several samples."""

    REASONS = {"hw_slowdown": 0x8, "sw_thermal_slowdown": 0x20, "hw_thermal_slowdown": 0x40, "sw_power_cap": 0x4}
    PERIOD_S = 0.002

    def __init__(self, device):
        self.device = device
        self.samples, self.max_mhz = [], None
        self.begin = 0
        self.stop_flag = threading.Event()
        self.ready = threading.Event()
        self.t = None
        self.err = None

    def _handle(self):
        import pynvml
        pynvml.nvmlInit()
        try:
            import torch
            pr = torch.cuda.get_device_properties(self.device)
            bus = f"{pr.pci_domain_id:08x}:{pr.pci_bus_id:02x}:{pr.pci_device_id:02x}.0"
            return pynvml.nvmlDeviceGetHandleByPciBusId(bus.encode())
        except Exception:
            return pynvml.nvmlDeviceGetHandleByIndex(self.device)

    def _run(self):
        try:
            import pynvml
            h = self._handle()
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(h, pynvml.NVML_CLOCK_SM)
            reasons = getattr(pynvml, "nvmlDeviceGetCurrentClocksEventReasons", None) or \
                pynvml.nvmlDeviceGetCurrentClocksThrottleReasons
            while not self.stop_flag.is_set():
                self.samples.append((pynvml.nvmlDeviceGetClockInfo(h, pynvml.NVML_CLOCK_SM), int(reasons(h))))
                self.ready.set()
                time.sleep(self.PERIOD_S)
        except Exception as e:  # NVML missing or refused: report it
            self.err = f"{type(e).__name__}: {e}"
        finally:
            self.ready.set()

    def start(self):
        self.t = threading.Thread(target=self._run, daemon=True)
        self.t.start()
        self.ready.wait(timeout=10)

    def mark(self):
        self.begin = len(self.samples)

    def stop(self):
        self.stop_flag.set()
        if self.t:
            self.t.join(timeout=5)
        taken = self.samples[self.begin:] or self.samples[-1:]
        if self.err or not taken:
            return {"sm_mhz": None, "sm_max_mhz": self.max_mhz, "reasons": [self.err or "no samples"], "samples": 0}
        mask = 0
        for _, m in taken:
            mask |= m
        reasons = sorted(k for k, bit in self.REASONS.items() if mask & bit)
        return {"sm_mhz": statistics.median(mhz for mhz, _ in taken), "sm_max_mhz": self.max_mhz, "reasons": reasons,
                "samples": len(taken), "source": "NVML every 2 ms during the timed region"}


def _rand_residues(torch, shape, moduli, gen):
    """uint64 residues (stored as int64) uniform modulo moduli[l] along axis -2 (two launches)."""
    # q < 2^61: 62 random bits reduced mod q (negligible bias for a benchmark input)
    x = torch.randint(0, 2 ** 62, shape, dtype=torch.int64, device="cuda", generator=gen)
    q = torch.tensor(moduli, dtype=torch.int64, device="cuda").view(len(moduli), 1)
    return torch.remainder(x, q)


def run_b200(args, rank, world):
    import torch
    import ckks_step
    import tb_capi

    dev = int(os.environ.get("LOCAL_RANK", 0))
    torch.cuda.set_device(dev)
    lib = tb_capi.lib()
    arr = (ctypes.c_int * len(BITS))(*BITS)
    mods = (ctypes.c_uint64 * len(BITS))()
    tb_capi.check(lib.tb_coeff_modulus_create(ctypes.c_uint64(N), arr, len(BITS), mods))
    moduli = [int(m) for m in mods]
    ctx = tb_capi.Context(tb_capi.SCHEME_CKKS, N, moduli)
    K = len(moduli)
    L = K - 1
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1234 + rank)
    stream = torch.cuda.current_stream()

    # keys: relinearization key and 13 Galois keys, key level [K-1][2][K][N]
    rlk = _rand_residues(torch, (K - 1, 2, K, N), moduli, gen)
    elts = []
    for k in STEPS_K:
        e = ctypes.c_uint32()
        ctx("galois_elt_from_step", k, ctypes.byref(e))
        elts.append(e.value)
    gks = [_rand_residues(torch, (K - 1, 2, K, N), moduli, gen) for _ in STEPS_K]
    # operands
    A = _rand_residues(torch, (PAIRS, 2, L, N), moduli[:L], gen)
    B = _rand_residues(torch, (PAIRS, 2, L, N), moduli[:L], gen)
    O = torch.empty((PAIRS, 2, L - 1, N), dtype=torch.int64, device="cuda")
    # the step's batch as SUB concurrent sub-batches, one stream each (SUB = 1: the whole
    # batch on the caller's stream): one sub-batch's short launches and wave tails
    # overlap the other's. Inside a sub-batch the pairs of each rotation step are
    # consecutive, so one grouped Galois call serves all 13 keys.
    SUB = args.streams if args.streams >= 1 and PAIRS % args.streams == 0 else 1
    stepper = ckks_step.BatchedCkksStep(torch, ctx, L, N, PAIRS, rlk, elts, gks, SUB)
    T3 = stepper.T3
    R = stepper.R

    def step(a, b, out, st=stream, sub=None):
        stepper(a, b, out, st, sub)

    def barrier():
        if world > 1:
            import torch.distributed as dist
            dist.barrier()
        torch.cuda.synchronize()

    if args.ks_persistent:
        lib.tb_keyswitch_set_persistent(1)
    # the autotuner times this step under each setting of the library's speed knobs
    # (NTT launch variants, key-switch budget; all compute identical words) and keeps
    # the fastest
    import tuning
    tuned = "off" if args.no_tune else tuning.tune_step(lambda: step(A, B, O), 14, stream)
    for _ in range(args.warmup):
        step(A, B, O)
    barrier()
    graph = None
    if args.graph:
        # the whole step (sub-batches, fork and join) captured once as a CUDA graph: the
        # library builds its per-element tables during the warm-up steps, and its
        # stream-ordered scratch allocations become graph memory nodes
        graph = torch.cuda.CUDAGraph()
        cap = torch.cuda.Stream()
        cap.wait_stream(stream)
        with torch.cuda.graph(graph, stream=cap, capture_error_mode="relaxed"):
            step(A, B, O, st=cap)
        stream.wait_stream(cap)
        for _ in range(args.warmup):
            graph.replay()
        barrier()
    clocks = ClockSampler(dev)
    clocks.start()
    if not graph:
        lib.tb_trace_enable(1)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.nvtx.range_push("timed")
    clocks.mark()
    e0.record(stream)
    for _ in range(args.steps):
        if graph:
            graph.replay()
        else:
            step(A, B, O)
    e1.record(stream)
    torch.cuda.nvtx.range_pop()
    barrier()
    ms = e0.elapsed_time(e1) / args.steps
    clk = clocks.stop()
    entries = (tb_capi_trace_entry * 64)()
    cnt = ctypes.c_int()
    if graph:
        # the graph replays the launches of one eager step: count them on one, traced
        lib.tb_trace_enable(1)
        step(A, B, O)
        barrier()
        tb_capi.check(lib.tb_trace_collect(entries, 64, ctypes.byref(cnt)))
        lib.tb_trace_enable(0)
        launches = sum(int(entries[i].launches) for i in range(cnt.value))
        trace = None
    else:
        tb_capi.check(lib.tb_trace_collect(entries, 64, ctypes.byref(cnt)))
        lib.tb_trace_enable(0)
        trace = {entries[i].name.decode(): (int(entries[i].launches), float(entries[i].total_ms))
                 for i in range(cnt.value)}
        launches = sum(v[0] for v in trace.values()) // args.steps
    if SUB > 1 or graph:
        # kernels of concurrent sub-batches share the GPU, so their event times say
        # nothing about one kernel: the per-kernel table and the roofline come from the
        # same step as one batch on one stream (kernels alone on the GPU), timed apart
        lib.tb_trace_enable(1)
        for _ in range(args.steps):
            step(A, B, O, sub=1)
        torch.cuda.synchronize()
        tb_capi.check(lib.tb_trace_collect(entries, 64, ctypes.byref(cnt)))
        lib.tb_trace_enable(0)
        trace = {entries[i].name.decode(): (int(entries[i].launches), float(entries[i].total_ms))
                 for i in range(cnt.value)}

    # plain per-op form: one ciphertext pair per call chain (batch 1), the way the
    # reference evaluator is driven (one multiply / relinearize / rescale / rotate call
    # per ciphertext); same kernels, same keys
    def per_op_chain(i):
        g = i % len(STEPS_K)
        ctx("multiply", L, A[i:i + 1], 0, B[i:i + 1], 0, T3[0:1], 0, 1, stream)
        ctx("relinearize", L, T3[0:1], 0, rlk, 1, stream)
        ctx("rescale_to_next", L, T3[0:1], 3 * L * N, R[0:1], 0, 2, 1, stream)
        ctx("apply_galois", L - 1, elts[g], R[0:1], 0, O[i:i + 1], 0, gks[g], 1, stream)

    per_op_pairs = min(PAIRS, PER_OP_PAIRS)
    for i in range(2):
        per_op_chain(i)
    barrier()
    e0.record(stream)
    for i in range(per_op_pairs):
        per_op_chain(i)
    e1.record(stream)
    barrier()
    per_op_ms = e0.elapsed_time(e1) / per_op_pairs

    # End to end through the C ABI with host buffers: every step copies its inputs in
    # from page-locked host memory and its results back out. Each step's batch runs as
    # --e2e-chunks sub-batches, the unit of the copy pipeline: the copies run on their own
    # streams (one per direction) with two device buffer sets, so a sub-batch's inputs
    # arrive while the one before computes and the one before that leaves; events order
    # each buffer's reuse. Every pair keeps the rotation step of the batched path.
    ech = args.e2e_chunks
    CH = ech if ech >= 1 and PAIRS % ech == 0 and PAIRS // ech >= len(STEPS_K) else 1
    PC = PAIRS // CH
    chunk_runs = [stepper.runs(c * PC, PC) for c in range(CH)]

    def chunk_step(c, j, a, b, out, st):
        # chunks on compute stream j use the step's scratch rows j*PC .. (j+1)*PC - 1
        stepper.chain(chunk_runs[c], PC, slice(j * PC, (j + 1) * PC), a, b, out, st)

    hA = torch.empty(A.shape, dtype=torch.int64, pin_memory=True)
    hB = torch.empty(B.shape, dtype=torch.int64, pin_memory=True)
    hO = [torch.empty(O.shape, dtype=torch.int64, pin_memory=True) for _ in range(2)]
    hA.copy_(A)
    hB.copy_(B)
    NBUF = 3   # device buffer sets: a chunk's copy-in need not wait for the compute two chunks back
    dA = [torch.empty_like(A[:PC]) for _ in range(NBUF)]
    dB = [torch.empty_like(B[:PC]) for _ in range(NBUF)]
    dO = [torch.empty_like(O[:PC]) for _ in range(NBUF)]
    s_in, s_out = torch.cuda.Stream(), torch.cuda.Stream()
    # two compute streams: unit u computes on s_comp[u % 2] (with the step's scratch rows
    # of that stream), so one chunk's short launches overlap the next chunk's, as the
    # sub-batches of the step do; its buffers are set u % NBUF
    # (one compute stream when the step's scratch rows cannot hold two chunks)
    NCS = 2 if 2 * PC <= PAIRS else 1
    s_comp = [torch.cuda.Stream() for _ in range(NCS)]
    ev = lambda: torch.cuda.Event()
    pending = {}

    # seed-compressed inputs (the reference GPU path's wire form of a symmetric
    # encryption: c0 and a 64-bit seed; c1 is regenerated from the seed on the device)
    hA0 = torch.empty((PAIRS, L, N), dtype=torch.int64, pin_memory=True)
    hB0 = torch.empty((PAIRS, L, N), dtype=torch.int64, pin_memory=True)
    hA0.copy_(A[:, 0])
    hB0.copy_(B[:, 0])
    hSA = torch.arange(1, PAIRS + 1, dtype=torch.int64).mul_(7919).add_(1 << 40).pin_memory()
    hSB = torch.arange(1, PAIRS + 1, dtype=torch.int64).mul_(104729).add_(1 << 41).pin_memory()
    dSA = [torch.empty((PC,), dtype=torch.int64, device="cuda") for _ in range(NBUF)]
    dSB = [torch.empty((PC,), dtype=torch.int64, device="cuda") for _ in range(NBUF)]
    seeded = {"on": False}

    def e2e_unit(u, k, c):
        j, sc = u % NBUF, u % NCS
        rows = slice(c * PC, (c + 1) * PC)
        arrived, computed, left = ev(), ev(), ev()
        with torch.cuda.stream(s_in):
            if ("computed", u - NBUF) in pending:
                s_in.wait_event(pending.pop(("computed", u - NBUF)))  # unit u-NBUF done reading dA[j], dB[j]
            if seeded["on"]:
                dA[j][:, 0].copy_(hA0[rows], non_blocking=True)
                dB[j][:, 0].copy_(hB0[rows], non_blocking=True)
                dSA[j].copy_(hSA[rows], non_blocking=True)
                dSB[j].copy_(hSB[rows], non_blocking=True)
            else:
                dA[j].copy_(hA[rows], non_blocking=True)
                dB[j].copy_(hB[rows], non_blocking=True)
            arrived.record(s_in)
        cs = s_comp[sc]
        cs.wait_event(arrived)
        if ("left", u - NBUF) in pending:
            cs.wait_event(pending.pop(("left", u - NBUF)))           # dO[j] read out
        if seeded["on"]:
            ctx("expand_seeded_batch", L, dSA[j], PC, 0, dA[j][:, 1], 2 * L * N, cs)
            ctx("expand_seeded_batch", L, dSB[j], PC, 0, dB[j][:, 1], 2 * L * N, cs)
        chunk_step(c, sc, dA[j], dB[j], dO[j], cs)
        computed.record(cs)
        with torch.cuda.stream(s_out):
            s_out.wait_event(computed)
            hO[k % 2][rows].copy_(dO[j], non_blocking=True)
            left.record(s_out)
        pending[("computed", u)] = computed
        pending[("left", u)] = left

    def e2e_run(first, count):
        start = ev()
        start.record(stream)            # the copy and compute streams begin after the timed start
        for st in (s_in, s_out, *s_comp):
            st.wait_event(start)
        for k in range(first, first + count):
            for c in range(CH):
                e2e_unit(k * CH + c, k, c)
        for key in [key for key in pending if key[0] == "left"]:
            stream.wait_event(pending[key])                          # every result is on the host
        pending.clear()

    e2e_run(0, max(1, args.warmup))
    barrier()
    e0.record(stream)
    e2e_run(0, args.steps)
    e1.record(stream)
    barrier()
    e2e_ms = e0.elapsed_time(e1) / args.steps
    # the host results of the last step equal the words of the same chunks computed on
    # the device from the resident inputs, one after another on one stream
    check = torch.empty_like(O)
    for c in range(CH):
        rows = slice(c * PC, (c + 1) * PC)
        chunk_step(c, 0, A[rows], B[rows], check[rows], stream)
    torch.cuda.synchronize()
    if not torch.equal(hO[(args.steps - 1) % 2], check.cpu()):
        raise RuntimeError("end-to-end results differ from the device-resident chunks' words")
    del check

    # the same pipeline when the inputs arrive seed-compressed: half the input bytes
    seeded["on"] = True
    e2e_run(0, max(1, args.warmup))
    barrier()
    e0.record(stream)
    e2e_run(0, args.steps)
    e1.record(stream)
    barrier()
    e2e_seeded_ms = e0.elapsed_time(e1) / args.steps
    seeded["on"] = False

    ms, e2e_ms, per_op_ms, e2e_seeded_ms = max_over_ranks([ms, e2e_ms, per_op_ms, e2e_seeded_ms], world, "cuda")
    return {"tuned": tuned, "e2e_seeded_ms": e2e_seeded_ms,
            "h2d_seeded": (hA0.numel() + hB0.numel() + hSA.numel() + hSB.numel()) * 8,
            "ms": ms, "e2e_ms": e2e_ms, "per_op_ms": per_op_ms, "per_op_pairs": per_op_pairs, "trace": trace, "launches": launches, "clocks": clk,
            "h2d": (A.numel() + B.numel()) * 8, "d2h": O.numel() * 8, "L": L, "K": K, "e2e_chunks": CH,
            "butterfly_rates": {"harvey": butterfly_rate(lib, moduli[0]),
                                "slack": butterfly_rate(lib, moduli[0], "slack"),
                                "wide": butterfly_rate(lib, moduli[0], "wide"),
                                "fp64": butterfly_rate(lib, min(moduli), "fp64")},
            "mul64": mul64_rates(lib),
            "butterfly_mix": butterfly_mix(moduli, L, N.bit_length() - 1), "sub": SUB}


def run_ntt_sweep(batch=256, reps=10):
    """The raw transform workload: `batch` polynomials x 8 limbs of 50-bit primes,
    N in {4096, ..., 32768}: forward NTT, dyadic product of pairs, inverse NTT.
    Algorithmic bytes: 16 N B L per transform (read + write), 24 N B L per dyadic
    product; GB/s and the fraction of the measured copy peak per kernel, and for the
    transforms the fraction of the arithmetic ceiling of the form they run, exact FP64
    for these moduli: (N/2) log2 N butterflies per limb over
    tb_measure_fp64_butterfly_rate."""
    import torch
    import tb_capi

    lib = tb_capi.lib()
    peak, _ = _peak_hbm()
    stream = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(8)
    out = {}
    ceiling = None
    for logn in (12, 13, 14, 15):
        n = 1 << logn
        arr = (ctypes.c_int * 8)(*([50] * 8))
        mods = (ctypes.c_uint64 * 8)()
        tb_capi.check(lib.tb_coeff_modulus_create(ctypes.c_uint64(n), arr, 8, mods))
        moduli = [int(m) for m in mods]
        if ceiling is None:
            ceiling = butterfly_rate(lib, moduli[0], "fp64")
        ctx = tb_capi.Context(tb_capi.SCHEME_RAW, n, moduli)
        x = _rand_residues(torch, (batch, 8, n), moduli, gen)
        y = _rand_residues(torch, (batch, 8, n), moduli, gen)
        z = torch.empty_like(x)

        def timed(fn):
            fn()
            torch.cuda.synchronize()
            e0.record(stream)
            for _ in range(reps):
                fn()
            e1.record(stream)
            torch.cuda.synchronize()
            return e0.elapsed_time(e1) / reps

        # the autotuner picks the launch variant per direction for this degree (restored
        # afterwards, so the sweep leaves the other workloads' choices alone)
        saved = []
        for fwd in (1, 0):
            v = ctypes.c_int(0)
            lib.tb_ntt_get_variant(fwd, min(logn, 14), ctypes.byref(v))
            saved.append(v.value)
        vf, vi = ctypes.c_int(0), ctypes.c_int(0)
        ctx("autotune_ntt", batch * 8, stream, ctypes.byref(vf), ctypes.byref(vi))
        words = batch * 8 * n
        ms_f = timed(lambda: ctx("ntt_forward", x, x, batch, 0, 8, 0, stream))
        ms_d = timed(lambda: ctx("dyadic_product", x, y, z, batch, 0, 8, stream))
        ms_i = timed(lambda: ctx("ntt_inverse", z, z, batch, 0, 8, 0, stream))
        row = {}
        for name, ms, bytes_ in (("ntt_forward", ms_f, 16 * words), ("dyadic", ms_d, 24 * words),
                                 ("ntt_inverse", ms_i, 16 * words)):
            gbs = bytes_ / (ms * 1e-3) / 1e9
            row[name] = {"ms": round(ms, 4), "GBps": round(gbs, 1), "frac_of_measured_hbm": round(gbs / peak, 4)}
            if name != "dyadic":   # (N/2) log2 N butterflies per limb
                rate = batch * 8 * (n // 2) * logn / (ms * 1e-3)
                row[name]["frac_of_fp64_ceiling"] = round(rate / ceiling, 4)
        row["variants"] = {"forward": vf.value, "inverse": vi.value}
        out[f"N={n}"] = row
        for fwd, v in zip((1, 0), saved):
            lib.tb_ntt_set_variant(fwd, min(logn, 14), v)
        del x, y, z
        ctx.close()
    return {"workload": f"{batch} polynomials x 8 limbs (50-bit primes)",
            "fp64_ceiling_gbutterflies_per_s": round(ceiling / 1e9, 2), "results": out}


UNEVEN_SHAPES = [(1, 4096, [36, 36, 37]), (3, 8192, [43, 43, 44, 44, 44]), (1, 16384, [48] * 9)]


def run_uneven(total=512, reps=5):
    """The uneven-batch workload: `total` ciphertext pairs whose ring degree is drawn from
    {4096, 8192, 16384} (3 / 5 / 9 primes; BFV, BGV, BFV), multiply -> relinearize ->
    rotate_rows(1), seeded uniform residues as ciphertexts and keys. Reports ops/s of
    the captured CUDA graph (one launch per batch), of the stream-overlapped calls and
    of the one-ciphertext-per-call path (each the best of three timings), and of the
    reference's own CUDA path one pair per call at the same shapes and counts."""
    import numpy as np
    import torch
    import tb_capi
    from uneven import ShapeGroup, UnevenBatch

    rng = np.random.default_rng(4096)
    draws = rng.integers(0, len(UNEVEN_SHAPES), total)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(99)
    lib = tb_capi.lib()
    groups, shapes = [], []
    for gi, (scheme, n, bits) in enumerate(UNEVEN_SHAPES):
        arr = (ctypes.c_int * len(bits))(*bits)
        mods = (ctypes.c_uint64 * len(bits))()
        tb_capi.check(lib.tb_coeff_modulus_create(ctypes.c_uint64(n), arr, len(bits), mods))
        moduli = [int(m) for m in mods]
        tmod = ctypes.c_uint64()
        tb_capi.check(lib.tb_plain_modulus_batching(ctypes.c_uint64(16384), 20, ctypes.byref(tmod)))
        ctx = tb_capi.Context(scheme, n, moduli, tmod.value)
        K, L, cnt = len(moduli), len(moduli) - 1, int((draws == gi).sum())
        shapes.append((scheme, n, moduli, tmod.value, cnt))
        e = ctypes.c_uint32()
        ctx("galois_elt_from_step", 1, ctypes.byref(e))
        groups.append(ShapeGroup(ctx, L, _rand_residues(torch, (cnt, 2, L, n), moduli[:L], gen),
                                 _rand_residues(torch, (cnt, 2, L, n), moduli[:L], gen),
                                 _rand_residues(torch, (K - 1, 2, K, n), moduli, gen),
                                 _rand_residues(torch, (K - 1, 2, K, n), moduli, gen), e.value))
    batch = UnevenBatch(groups)
    stream = torch.cuda.current_stream()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)

    def timed(fn, k, warm=2, trials=3):
        """Best of `trials` timings of k calls, after `warm` untimed calls (the first calls
        of a mode grow its streams' pools and build its tables)."""
        for _ in range(warm):
            fn()
        torch.cuda.synchronize()
        best = float("inf")
        for _ in range(trials):
            e0.record(stream)
            for _ in range(k):
                fn()
            e1.record(stream)
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1) / k)
        return best

    ms_streams = timed(batch.run, reps)
    ms_per_op = timed(batch.run_per_op, 1)
    batch.capture()
    ms_graph = timed(batch.replay, reps)
    # the same batch with every group's key switches in one persistent launch per step
    shaped = UnevenBatch(groups)
    shaped.set_shapes(True)
    ms_shapes = timed(shaped.run, reps)
    shaped.capture()
    ms_shapes_graph = timed(shaped.replay, reps)
    best = min(ms_graph, ms_shapes_graph)
    out = {"workload": "uneven_bfv_bgv_n4096_8192_16384_mul_relin_rotate", "ciphertexts": total,
           "groups": {f"N={g.ctx.n},L={g.L}": g.count for g in groups},
           "graph_ops_per_s": round(total / (ms_graph * 1e-3), 1),
           "streams_ops_per_s": round(total / (ms_streams * 1e-3), 1),
           "shapes_ops_per_s": round(total / (ms_shapes * 1e-3), 1),
           "shapes_graph_ops_per_s": round(total / (ms_shapes_graph * 1e-3), 1),
           "per_op_ops_per_s": round(total / (ms_per_op * 1e-3), 1),
           "graph_over_per_op": round(ms_per_op / best, 2)}
    ref = reference_gpu_uneven(shapes)
    if ref is not None:
        out["reference_gpu_per_op"] = ref
        if "ms_per_batch" in ref:
            out["graph_over_reference_gpu_per_op"] = round(ref["ms_per_batch"] / best, 2)
    return out


def _ref_gpu_uneven_worker(args):
    """Child process: the reference's CUDA evaluator one ciphertext pair per call at each
    shape of the uneven batch (ms per op, decrypted result checked)."""
    shapes, ops = args
    devnull = os.open(os.devnull, os.O_WRONLY)
    os.dup2(devnull, 1)
    lib = ctypes.CDLL(os.path.join(ROOT, "oracle", "_ref", "libtroyref_gpu.so"))
    lib.ref_gpu_batch_chain.argtypes = [ctypes.c_int, ctypes.c_size_t, ctypes.POINTER(ctypes.c_uint64), ctypes.c_int,
                                        ctypes.c_uint64, ctypes.c_int, ctypes.POINTER(ctypes.c_double),
                                        ctypes.POINTER(ctypes.c_int)]
    res = []
    for scheme, n, moduli, t, _ in shapes:
        arr = (ctypes.c_uint64 * len(moduli))(*moduli)
        ms, ok = ctypes.c_double(), ctypes.c_int()
        rc = lib.ref_gpu_batch_chain(scheme, n, arr, len(moduli), t, ops, ctypes.byref(ms), ctypes.byref(ok))
        res.append((rc, ms.value, ok.value))
    return res


def reference_gpu_uneven(shapes, ops=8):
    """The reference's own CUDA path on the uneven batch's chain (multiply, relinearize,
    rotate rows), one ciphertext pair per call, at each shape: the batch's time is each
    group's count times that shape's time per op. None when that library is not built."""
    if not os.path.exists(os.path.join(ROOT, "oracle", "_ref", "libtroyref_gpu.so")):
        return None
    with mp.get_context("spawn").Pool(1) as pool:
        res = pool.apply(_ref_gpu_uneven_worker, ((shapes, ops),))
    if any(rc == 1 or ms <= 0 for rc, ms, _ in res):
        return {"unavailable": "reference CUDA path raised an exception"}
    ms_batch = sum(cnt * ms for (_, _, _, _, cnt), (_, ms, _) in zip(shapes, res))
    total = sum(cnt for *_, cnt in shapes)
    return {"ops_per_s": round(total / (ms_batch * 1e-3), 1), "ms_per_batch": round(ms_batch, 3),
            "ms_per_op": {f"N={n}": round(ms, 3) for (_, n, *_), (_, ms, _) in zip(shapes, res)},
            "decrypts_correctly": all(ok == 1 for *_, ok in res),
            "form": "reference EvaluatorCuda compiled for sm_100a, one pair per call, "
                    f"{ops} ops per shape after 2 warm-up ops, in a child process"}


def _pinned(a):
    """A page-locked copy of a uint64 array (what a server's receive buffers would be)."""
    import numpy as np
    import torch
    t = torch.empty(a.size, dtype=torch.int64, pin_memory=True)
    out = t.numpy().view(np.uint64)
    out[:] = a
    _pinned.keep.append(t)
    return out


_pinned.keep = []


def run_serving(seconds_per_rate=2.0, max_requests=400, pool_size=32):
    """Poisson arrivals of encrypted vector x matrix requests (input dimension in
    {64, ..., 1024}, output in {16, ..., 256}, seeded) through MatmulServer at each rate
    of SERVE_RATES plus one burst with every request queued at once. Latency is
    arrival to completion on the host steady clock; throughput is completed requests
    over first arrival to last completion."""
    sys.path.insert(0, os.path.join(ROOT, "seal-cuda_b200", "lib"))
    import numpy as np
    import pytroy

    t = pytroy.PlainModulus.batching(SERVE_N, 20)
    p = pytroy.EncryptionParameters(pytroy.SchemeType.bfv)
    p.set_poly_modulus_degree(SERVE_N)
    p.set_coeff_modulus(pytroy.CoeffModulus.create(SERVE_N, SERVE_BITS))
    p.set_plain_modulus(t)
    ctx = pytroy.SEALContext(p)
    keygen = pytroy.KeyGenerator(ctx)
    enc = pytroy.BatchEncoder(ctx)
    encryptor = pytroy.Encryptor(ctx, keygen.create_public_key(), keygen.secret_key())
    rng = np.random.default_rng(2718)
    pool = []
    for _ in range(pool_size):
        inp, out = int(rng.integers(1, 17)) * 64, int(rng.integers(1, 17)) * 16
        x = rng.integers(0, t.value(), inp, dtype=np.uint64)
        w = rng.integers(0, t.value(), inp * out, dtype=np.uint64)
        h = pytroy.MatmulHelper(1, inp, out, SERVE_N)
        cts = h.encrypt_inputs(encryptor, enc, x)
        words = np.concatenate([np.asarray(c.data(), np.uint64) for c in cts[0]])
        # page-locked request and result buffers, as a server's receive/send buffers;
        # requests sharing a pool entry overwrite its result buffer (values not read here)
        blocks = (out + h.output_block - 1) // h.output_block
        res = _pinned(np.zeros(blocks * 2 * (len(SERVE_BITS) - 1) * SERVE_N, np.uint64))
        pool.append((inp, out, _pinned(words), _pinned(w), res))
    server = pytroy.MatmulServer(ctx, memory_budget=16 << 30, slots=3)
    now = pytroy.MatmulServer.now
    for r in pool[:8]:  # warm-up
        server.submit(r[0], r[1], r[2], r[3], now(), outputs=r[4])
    server.drain(60.0)

    def run(rate):
        count = max_requests if rate is None else max(20, min(max_requests, int(rate * seconds_per_rate)))
        gaps = np.zeros(count) if rate is None else rng.exponential(1.0 / rate, count)
        start = now()
        due = start + np.cumsum(gaps)
        ids, k = [], 0
        st0 = server.stats()
        waves0 = st0["waves"]
        while k < count or not server.idle():
            tnow = now()
            while k < count and due[k] <= tnow:
                r = pool[k % len(pool)]
                ids.append(server.submit(r[0], r[1], r[2], r[3], float(due[k]), outputs=r[4]))
                k += 1
            server.step()
            if tnow - start > 120.0:
                raise RuntimeError("serving run did not finish")
        lat, first, last, ok = [], None, None, 0
        for rid in ids:
            _, arrival, done, good = server.take(rid)
            ok += bool(good)
            lat.append(1e3 * (done - arrival))
            first = arrival if first is None else min(first, arrival)
            last = done if last is None else max(last, done)
        st = server.stats()
        waves = st["waves"] - waves0
        host = {k: round(st[k] - st0[k], 4) for k in ("launch_host_s", "alloc_host_s", "reap_host_s", "device_s")}
        return {"rate_rps": rate if rate is not None else "burst", "requests": count, "ok": ok,
                "p50_ms": round(float(np.percentile(lat, 50)), 3), "p99_ms": round(float(np.percentile(lat, 99)), 3),
                "throughput_rps": round(count / (last - first), 1), "mean_wave": round(count / max(1, waves), 2),
                "server_seconds": host}

    run(None)   # warm-up burst: the server's device pool grows to its largest wave once
    runs = [run(r) for r in SERVE_RATES] + [run(None)]
    return {"workload": "bfv_n8192_L4_matmul_poisson", "slots": 3, "memory_budget_gb": 16,
            "request_shapes": "in {64..1024} x out {16..256}, MatmulHelper coefficient encoding",
            "latency": "arrival to completion, host steady clock", "runs": runs}


def max_over_ranks(times_ms, world, device):
    """Each timing (ms) maxed over the ranks of the process group (identity for one
    rank): replicas run independently and the job is as slow as its slowest rank."""
    if world == 1:
        return list(times_ms)
    import torch
    import torch.distributed as dist
    t = torch.tensor(list(times_ms), dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return [float(x) for x in t]


def job_rate(units_per_rank, world, ms):
    """Whole-job throughput: the units all ranks processed over the slowest rank's time."""
    return units_per_rank * world / (ms * 1e-3)


class tb_capi_trace_entry(ctypes.Structure):
    _fields_ = [("name", ctypes.c_char * 32), ("launches", ctypes.c_uint64), ("total_ms", ctypes.c_double)]


def algorithmic_bytes_per_step(L):
    """Bytes each traced kernel must move per step at this workload (8-byte words):
    L data limbs at multiply/relinearize, L-1 after the rescale, K = L + 1 key limbs."""
    n, B, W = N, PAIRS, 8
    Lr = L - 1

    def ks(l):  # per key switch of one ciphertext at level l (CKKS)
        return {
            "ks_target_intt": 2 * l * n * W,
            "ks_modup_ntt": (l + l * l) * n * W,                     # each target limb in once, L*L digits out
            # digits of the l data moduli (l - 1 per modulus) + the target limb in,
            # 2 l accumulators out
            "ks_inner_product": (l * l + 2 * l) * n * W,
            # the l special-modulus digits in (inner product fused into the load), 2 rows out
            "ks_special_intt": (l + 2) * n * W,
            "ks_moddown": 2 * l * 4 * n * W,                         # last, acc, ct in; ct out
        }

    out = {"tensor": B * 7 * L * n * W,
           "rescale_last_intt": B * 2 * 2 * n * W,
           "rescale_ntt": B * 2 * Lr * 3 * n * W,
           "galois_permute": B * 5 * Lr * n * W}
    for name, v in ks(L).items():
        out[name] = B * v
    for name, v in ks(Lr).items():
        out[name] += B * v
    # keys are read once per launch: relinearization key + one Galois key per group; the
    # inner product reads their data-modulus columns, the special transform the last one
    out["ks_inner_product"] += 2 * L * L * n * W + len(STEPS_K) * 2 * Lr * Lr * n * W
    out["ks_special_intt"] += 2 * L * n * W + len(STEPS_K) * 2 * Lr * n * W
    return out


def roofline(res, steps):
    """Dominant kernel (most device time): algorithmic bytes per launch / mean launch time."""
    trace = res["trace"]
    alg = algorithmic_bytes_per_step(res["L"])
    peak, kind = _peak_hbm()
    table = {}
    traffic = measured_traffic()
    for name, (launches, total_ms) in trace.items():
        per_launch_ms = total_ms / launches
        b = alg.get(name)
        gbs = (b * steps / launches) / (per_launch_ms * 1e-3) / 1e9 if b else None
        table[name] = {"launches_per_step": launches // steps, "ms_per_step": round(total_ms / steps, 4),
                       "GBps": round(gbs, 1) if gbs else None, "frac_hbm": round(gbs / peak, 4) if gbs else None}
        if name in traffic:
            table[name]["traffic_per_launch"] = round(traffic[name] * steps / launches)
    name = max(trace.items(), key=lambda kv: kv[1][1])[0]
    launches, total_ms = trace[name]
    per_launch_ms = total_ms / launches
    bpl = alg[name] * steps / launches
    achieved = bpl / (per_launch_ms * 1e-3) / 1e9
    tr = measured_traffic().get(name)
    # the transforms against the arithmetic ceiling (butterflies per second): the rates of
    # the butterflies they run, weighted by the shares of each kind
    bfly = butterflies_per_step(res["L"])
    rates = res["butterfly_rates"]
    ceilings = {k: 1.0 / sum(sh / rates[kind] for kind, sh in mix.items()) for k, mix in res["butterfly_mix"].items()}
    for k, row in table.items():
        if k in bfly:
            row["arith_frac"] = round(bfly[k] / (row["ms_per_step"] * 1e-3) / ceilings[k], 4)
    # the roofline is stated against HBM (achieved / peak in GB/s); "limited_by" names the
    # resource the kernel uses the larger fraction of: HBM bandwidth, or the arithmetic
    # ceiling of the transforms ("arith" sub-object)
    rate = bfly[name] * steps / launches / (per_launch_ms * 1e-3) if name in bfly else None
    limited_by = "arith" if rate and rate / ceilings[name] > achieved / peak else "hbm"
    out = {"kernel": name, "bound": "hbm", "limited_by": limited_by, "achieved": round(achieved, 1), "peak": peak,
           "unit": "GB/s",
           "frac": round(achieved / peak, 4),
           "traffic": round(tr * steps / launches) if tr else None,
           "traffic_source": "ncu dram__bytes_read.sum + dram__bytes_write.sum of this kernel at this shape "
                             "(profiles/ckks_step_n16384_traffic.md), per launch" if tr else None,
           "algorithmic_bytes_per_launch": round(bpl),
           "peak_source": "of measured (MEASURED_PEAKS.json hbm_gbs)" if kind == "measured" else "of fallback",
           "kernels": table}
    if res.get("sub", 1) > 1:
        out["timing"] = (f"kernel times from the same {steps} steps run as one batch on one stream after the "
                         f"timed region (which runs {res['sub']} concurrent sub-batches)")
    if rate:
        mix, ceil = res["butterfly_mix"][name], ceilings[name]
        out["arith"] = {"achieved": round(rate / 1e9, 2), "peak": round(ceil / 1e9, 2), "unit": "Gbutterfly/s",
                        "frac": round(rate / ceil, 4),
                        "butterflies_per_launch": round(bfly[name] * steps / launches),
                        "peak_source": "measured here, operands in registers (tb_measure_*_butterfly_rate), weighted by "
                                       "the shares of the kernel's butterflies of each kind: "
                                       + ", ".join(f"{k} {sh:.4f} at {rates[k] / 1e9:.2f} G/s"
                                                   for k, sh in mix.items() if sh)}
        # the machine bound of an exact-quotient integer butterfly: its Shoup product is one
        # high and two low 64-bit products (the wide form estimates its quotient from 32-bit
        # products and may pass it; FP64 butterflies run on the FP64 pipe)
        m = res["mul64"]
        out["arith"]["integer_machine_bound"] = {
            "mul_lo_per_s": round(m["lo"] / 1e9, 1), "mul_hi_per_s": round(m["hi"] / 1e9, 1), "unit": "G/s",
            "butterflies_per_s": round(1.0 / (1.0 / m["hi"] + 2.0 / m["lo"]) / 1e9, 2),
            "source": "tb_measure_mul64_rate: mul.lo.u64 / mul.hi.u64 in independent chains; "
                      "bound = 1 / (1/hi + 2/lo) butterflies per second"}
    return out


def butterflies_per_step(L):
    """Butterflies each traced transform kernel runs per step: (N/2) log2 N per limb
    transformed; L data limbs at multiply/relinearize, L-1 after the rescale."""
    per = (N // 2) * (N.bit_length() - 1)
    B, Lr = PAIRS, L - 1
    limbs = {"ks_target_intt": L + Lr, "ks_modup_ntt": L * L + Lr * Lr, "ks_special_intt": 2 + 2,
             "ks_moddown": 2 * (L + Lr), "rescale_last_intt": 2, "rescale_ntt": 2 * Lr}
    return {k: B * v * per for k, v in limbs.items()}


def butterfly_rate(lib, q, kind="harvey"):
    """Butterflies per second of one of the library's butterflies with everything in
    registers: "harvey" the lazy integer one (tb_measure_butterfly_rate), "slack" the one
    without the conditional subtraction, "wide" the no-subtraction form's with the
    estimated quotient, "fp64" the exact FP64 one (moduli below 2^50)."""
    fn = {"harvey": lib.tb_measure_butterfly_rate, "slack": lib.tb_measure_slack_butterfly_rate,
          "wide": lib.tb_measure_wide_butterfly_rate, "fp64": lib.tb_measure_fp64_butterfly_rate}[kind]
    fn.argtypes = [ctypes.c_uint64, ctypes.c_void_p, ctypes.POINTER(ctypes.c_double)]
    r = ctypes.c_double(0)
    import tb_capi
    tb_capi.check(fn(q, None, ctypes.byref(r)))
    return r.value


def fwd_subtracting_stages(logn, M=16):
    """Stages of a forward transform of 2^logn coefficients with deferred reductions
    (bound M q; the library's fwd_bound / fwd_subtracts) that run the subtracting
    butterfly; the others run the slack one."""
    b, sub = 4, 0
    for _ in range(logn):
        if b + 2 <= M:
            b += 2
        else:
            b, sub = M // 2 + 2, sub + 1
    return sub


def mul64_rates(lib):
    """The device's 64-bit multiply throughputs (tb_measure_mul64_rate): products per
    second of mul.lo.u64 ("lo") and mul.hi.u64 ("hi")."""
    fn = lib.tb_measure_mul64_rate
    fn.argtypes = [ctypes.c_int, ctypes.c_void_p, ctypes.POINTER(ctypes.c_double)]
    out = {}
    import tb_capi
    for kind, key in ((0, "lo"), (1, "hi")):
        r = ctypes.c_double(0)
        tb_capi.check(fn(kind, None, ctypes.byref(r)))
        out[key] = r.value
    return out


def butterfly_mix(moduli, L, logn):
    """Per transform kernel at the benchmark shape, the shares of its butterflies of each
    kind: "fp64" (limbs of moduli below 2^50, N = 4096 .. 32768), and in integer form "wide"
    (no subtraction, estimated quotient: moduli below 2^57, in the mod-up at most 15
    digits), "slack" (the non-subtracting stages of the deferred-reduction form, moduli
    below 2^60) and "harvey" (its subtracting stages, every stage above 2^60, and the
    inverse transforms). The mod-up covers digit j on every key modulus but its own at L
    data limbs and at L-1 after the rescale; the mod-down, the rescale and the target
    inverse transform data limbs, the special and last-limb inverses one limb each."""
    special = moduli[-1]
    sub = fwd_subtracting_stages(logn) / logn

    def kinds(q, wide=True, forward=True):
        if q < (1 << 50) and 12 <= logn <= 15:
            return {"fp64": 1.0}
        if forward and wide and q < (1 << 57):
            return {"wide": 1.0}
        if forward and q < (1 << 60):
            return {"slack": 1.0 - sub, "harvey": sub}
        return {"harvey": 1.0}

    def mean(rows):
        return {k: sum(r.get(k, 0.0) for r in rows) / len(rows) for k in ("fp64", "wide", "slack", "harvey")}

    up = []
    for lv in (L, L - 1):
        targets = list(moduli[:lv]) + [special]
        up += [kinds(q, lv <= 15) for j in range(lv) for i, q in enumerate(targets) if i != j]
    data = [q for lv in (L, L - 1) for q in moduli[:lv]]
    return {"ks_modup_ntt": mean(up), "ks_moddown": mean([kinds(q) for q in data]),
            "rescale_ntt": mean([kinds(q) for q in moduli[:L - 1]]),
            "ks_target_intt": mean([kinds(q, forward=False) for q in data]),
            "ks_special_intt": mean([kinds(special, forward=False)]),
            "rescale_last_intt": mean([kinds(moduli[L - 1], forward=False)])}


TRAFFIC_PROFILE = os.path.join(ROOT, "profiles", "ckks_step_n16384_traffic.md")


def measured_traffic():
    """DRAM bytes (read + write) per step of each kernel of the one-stream step at the
    benchmark's shape (64 pairs, L = 8 and 7), from the ncu capture summarised in
    profiles/ckks_step_n16384_traffic.md (its json block: kernel -> bytes per step);
    {} when the summary is absent."""
    try:
        with open(TRAFFIC_PROFILE) as f:
            text = f.read()
        block = text.split("```json", 1)[1].split("```", 1)[0]
        return {k: float(v) for k, v in json.loads(block)["bytes_per_step"].items()}
    except (OSError, IndexError, KeyError, ValueError):
        return {}


# -------------------------------------------------------------- CPU baseline
def _ref_worker(args):
    """One process: a reference session at the benchmark parameters, `ops` timed ops."""
    ops, seed = args
    import numpy as np
    from oracle import RefSession

    sys.path.insert(0, os.path.join(ROOT, "oracle"))
    import ctypes as C
    lib = C.CDLL(os.path.join(ROOT, "oracle", "_ref", "libtroyref.so"))
    moduli = _ref_moduli()
    s = RefSession(2, N, moduli, 0, np.arange(seed, seed + 8, dtype=np.uint64))
    rng = np.random.default_rng(seed)
    v = rng.uniform(-1, 1, N // 2) + 1j * rng.uniform(-1, 1, N // 2)
    w = rng.uniform(-1, 1, N // 2) + 1j * rng.uniform(-1, 1, N // 2)
    a, b = s.encrypt_ckks(v, 2.0 ** SCALE_BITS), s.encrypt_ckks(w, 2.0 ** SCALE_BITS)
    lib.ref_ct_free.argtypes = [C.c_void_p, C.c_int]
    # warm: create the relinearization key and the Galois keys this worker uses
    ks = [STEPS_K[(seed + i) % len(STEPS_K)] for i in range(ops)]
    m = s.multiply(a, b)
    r = s.relinearize(m)
    rs = s.rescale(r)
    for k in set(ks):
        lib.ref_ct_free(s.h, s.rotate_vector(rs, k))
    t0 = time.perf_counter()
    for k in ks:
        m = s.multiply(a, b)
        r = s.relinearize(m)
        rs = s.rescale(r)
        o = s.rotate_vector(rs, k)
        for x in (m, r, rs, o):
            lib.ref_ct_free(s.h, x)
    return ops, time.perf_counter() - t0


def _ref_moduli():
    from oracle import Oracle
    return Oracle("ref").coeff_modulus_create(N, BITS)


def cpu_reference(ops_per_worker, workers):
    """ops/s of the reference CPU path, one independent session per process."""
    ctxm = mp.get_context("spawn")
    with ctxm.Pool(workers) as pool:
        t0 = time.perf_counter()
        res = pool.map(_ref_worker, [(ops_per_worker, 17 + 97 * i) for i in range(workers)])
        wall = time.perf_counter() - t0
    ops = sum(r[0] for r in res)
    busy = max(r[1] for r in res)
    return ops / busy, ops, busy, wall


def _ref_gpu_worker(args):
    """Child process: the reference's own CUDA evaluator (oracle/_ref/libtroyref_gpu.so)
    one pair per call; its stdout prints are discarded."""
    ops, = args
    devnull = os.open(os.devnull, os.O_WRONLY)
    os.dup2(devnull, 1)
    lib = ctypes.CDLL(os.path.join(ROOT, "oracle", "_ref", "libtroyref_gpu.so"))
    lib.ref_gpu_ckks_chain.argtypes = [ctypes.c_size_t, ctypes.POINTER(ctypes.c_uint64), ctypes.c_int, ctypes.c_int,
                                       ctypes.c_int, ctypes.POINTER(ctypes.c_int), ctypes.c_int,
                                       ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_double)]
    moduli = _ref_moduli()
    arr = (ctypes.c_uint64 * len(moduli))(*moduli)
    st = (ctypes.c_int * len(STEPS_K))(*STEPS_K)
    ms, err = ctypes.c_double(), ctypes.c_double()
    rc = lib.ref_gpu_ckks_chain(N, arr, len(moduli), SCALE_BITS, ops, st, len(STEPS_K), ctypes.byref(ms),
                                ctypes.byref(err))
    return rc, ms.value, err.value


def reference_gpu_per_op(ops=16):
    """ops/s of the reference's CUDA path (compiled for sm_100a from its sources by
    oracle/Makefile) on this workload, one pair per call chain, as the reference is
    used; None when that library is not built."""
    if not os.path.exists(os.path.join(ROOT, "oracle", "_ref", "libtroyref_gpu.so")):
        return None
    with mp.get_context("spawn").Pool(1) as pool:
        rc, ms, err = pool.apply(_ref_gpu_worker, ((ops,),))
    if rc == 1 or ms <= 0:
        return {"unavailable": "reference CUDA path raised an exception"}
    return {"value": round(1e3 / ms, 2), "unit": "ops/s", "ms_per_op": round(ms, 3), "ops": ops,
            "max_abs_error_vs_fp64": err,
            "note": "reference EvaluatorCuda compiled for sm_100a; pending CUDA error after the run" if rc == 2
            else "reference EvaluatorCuda compiled for sm_100a"}


def _cpu_model():
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                if line.startswith("model name"):
                    return line.split(":", 1)[1].strip()
    except OSError:
        pass
    import platform
    return platform.processor() or "unknown"


def _cpu_count():
    try:
        return len(os.sched_getaffinity(0))
    except Exception:
        return os.cpu_count() or 1


# ---------------------------------------------------------------------- main
def main():
    global PAIRS
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--cpu-ops", type=int, default=32, help="ops per CPU worker per step of --impl reference")
    ap.add_argument("--cpu-baseline-ops", type=int, default=320,
                    help="ops per CPU worker in the cpu_baseline sample of the GPU arm (about 10 - 20 s)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-serving", action="store_true", help="skip the serving-loop measurement")
    ap.add_argument("--no-uneven", action="store_true", help="skip the uneven-batch measurement")
    ap.add_argument("--no-ntt-sweep", action="store_true", help="skip the raw transform sweep")
    ap.add_argument("--no-reference-gpu", action="store_true", help="skip timing the reference CUDA path")
    ap.add_argument("--e2e-chunks", type=int, default=E2E_CHUNKS,
                    help="chunks per step of the end-to-end copy pipeline")
    ap.add_argument("--streams", type=int, default=HEADLINE_SUB_BATCHES,
                    help="concurrent sub-batches (one stream each) per step of the headline workload")
    ap.add_argument("--ks-persistent", action="store_true",
                    help="key switching through one persistent launch per step (tb_keyswitch_set_persistent)")
    ap.add_argument("--no-graph", dest="graph", action="store_false",
                    help="time the step as eager launches instead of one captured CUDA graph per step")
    ap.add_argument("--no-tune", action="store_true",
                    help="keep the default launch settings (for profiler captures: no tuning launches first)")
    ap.add_argument("--pairs", type=int, default=DEFAULT_PAIRS,
                    help="ciphertext pairs per step (smaller cases for profiling)")
    args = ap.parse_args()
    PAIRS = args.pairs
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    cores = _cpu_count()

    if args.impl == "reference":
        if rank != 0:
            return
        if not os.path.exists(os.path.join(ROOT, "oracle", "_ref", "libtroyref.so")):
            print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libtroyref.so is not built (it is "
                              "compiled from the reference's sources, which are not on this machine)"}))
            return
        workers = cores
        vals = []
        for i in range(args.warmup + args.steps):
            v, ops, busy, wall = cpu_reference(args.cpu_ops, workers)
            if i >= args.warmup:
                vals.append((v, ops, busy))
        value = sum(v[1] for v in vals) / sum(v[2] for v in vals)
        line = {"metric": METRIC, "value": round(value, 3), "unit": "ops/s", "impl": "reference",
                "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
                "ms_per_step": round(1e3 * statistics.mean(v[2] for v in vals), 3), "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "u64 (exact modular)", "data": "synthetic",
                "config": {"workload": WORKLOAD, "global_batch": args.cpu_ops * workers, "seq_len": N,
                           "parallelism": f"{workers} CPU processes"},
                "cpu_baseline": {"value": round(value, 3), "unit": "ops/s", "cores": workers, "kind": "reference",
                                 "cpu_model": _cpu_model(),
                                 "sample": f"{args.cpu_ops} ops per process x {workers} processes per step"},
                "e2e": {"value": round(value, 3), "unit": "ops/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
        print(json.dumps(line))
        return

    if world > 1:
        import datetime

        import torch
        import torch.distributed as dist
        torch.cuda.set_device(int(os.environ.get("LOCAL_RANK", 0)))
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    res = run_b200(args, rank, world)
    ops_total = PAIRS * world
    value = job_rate(PAIRS, world, res["ms"])
    e2e = job_rate(PAIRS, world, res["e2e_ms"])
    line = None
    if rank == 0:
        cpu = None
        if not args.no_cpu_baseline and os.path.exists(os.path.join(ROOT, "oracle", "_ref", "libtroyref.so")):
            workers = min(cores, 32)
            v, ops, busy, wall = cpu_reference(args.cpu_baseline_ops, workers)
            cpu = {"value": round(v, 3), "unit": "ops/s", "cores": workers, "kind": "reference",
                   "cpu_model": _cpu_model(),
                   "sample": f"{ops} ops ({args.cpu_baseline_ops} per process x {workers} processes), "
                             f"{busy:.1f} s"}
        per_op = 1e3 / res["per_op_ms"]
        ref_gpu = None if args.no_reference_gpu else reference_gpu_per_op()
        if ref_gpu and "value" in ref_gpu:
            ref_gpu["batched_over_reference_gpu_per_op"] = round(value / (ref_gpu["value"] * world), 2)
        serving = None if args.no_serving else run_serving()
        uneven = None if args.no_uneven else run_uneven()
        sweep = None if args.no_ntt_sweep else run_ntt_sweep()
        line = {"metric": METRIC, "value": round(value, 2), "unit": "ops/s", "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": round(res["ms"], 4), "higher_is_better": True,
                "scaling": "weak", "vs_baseline": None, "dtype": "u64 (exact modular)",
                "data": "synthetic: seeded uniform residues for ciphertexts and keys",
                "config": {"workload": WORKLOAD, "global_batch": ops_total, "seq_len": N,
                           "parallelism": "replicas" if world > 1 else "single GPU",
                           "l2": "inputs (256 MB) larger than L2", "tuned": res["tuned"],
                           "concurrent_sub_batches": res["sub"], "cuda_graph": bool(args.graph)},
                "e2e": {"value": round(e2e, 2), "unit": "ops/s", "h2d_bytes_per_step": res["h2d"],
                        "d2h_bytes_per_step": res["d2h"], "sub_batches_per_step": res["e2e_chunks"]},
                "e2e_seeded": {"value": round(job_rate(PAIRS, world, res["e2e_seeded_ms"]), 2), "unit": "ops/s",
                               "h2d_bytes_per_step": res["h2d_seeded"], "d2h_bytes_per_step": res["d2h"],
                               "form": "inputs as c0 plus a 64-bit seed (the reference GPU path's wire form of a "
                                       "symmetric encryption); c1 regenerated by cuRAND on the device inside the "
                                       "timed region (tb_expand_seeded_batch)"},
                "gpu_launches": res["launches"],
                "roofline": roofline(res, args.steps),
                "cpu_baseline": cpu,
                "plain_per_op": {"value": round(per_op * world, 2), "unit": "ops/s", "pairs": res["per_op_pairs"],
                                 "form": "one pair per call chain (batch 1), same kernels and keys",
                                 "batched_over_per_op": round(value / (per_op * world), 2)},
                "reference_gpu_per_op": ref_gpu,
                # the batching gains as top-level numbers: this library one pair per call,
                # and the reference's own CUDA evaluator one pair per call
                "plain_per_op_ops_per_s": round(per_op * world, 2),
                "reference_gpu_per_op_ops_per_s": ref_gpu.get("value") if ref_gpu else None,
                "batched_over_plain_per_op": round(value / (per_op * world), 2),
                "batched_over_reference_gpu_per_op": ref_gpu.get("batched_over_reference_gpu_per_op")
                if ref_gpu else None,
                "serving": serving,
                "uneven_batch": uneven,
                "ntt_sweep": sweep,
                "clocks": res["clocks"],
                "kernels_ms_per_step": {k: round(v[1] / args.steps, 4) for k, v in sorted(res["trace"].items())}}
        print(json.dumps(line))
    if world > 1:
        import torch.distributed as dist
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
