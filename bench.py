#!/usr/bin/env python
"""Benchmark of the group-then-align hot path on one GB300 (or N replicas).

Workload (one step): the device hot path over 200,000 synthetic DNA
sequences from 20,000 families (uniform roots 200-3000 nt, GC 0.45, members
with 1-10 % substitutions and 1 % indels of mean length 2, seed 2) at
identity 95 with 64 bands:
  sketch (64 minhash signatures per sequence) -> bucket (rep rows of 64
  bands) -> candidate pairs of all bands, deduplicated -> banded bit-parallel
  LCS of every distinct pair -> sorted unique edge list.
The packed database is resident in HBM before timing; L2 is flushed (256 MiB
write) before every timed step.  Leiden and the result file (host, unchanged
from the reference) are not part of the step.

metric  seqs clustered/s = sequences / step time (whole job, all ranks).
e2e     the same through ngia_ctx_run_host on pinned host buffers: H2D of the
        packed planes, offsets and lengths, the device path, D2H of the edges.
--impl reference   times the reference's own CPU implementation of the same
        path (makedb pack+sketch+group, buildGraph candidates+align+emit;
        the reference code built as a host OpenMP program) on a bounded
        sample of the workload with all host cores.
pairs   (one GPU) aligned cells/s of the batched aligner against the plain
        one-thread-per-pair form launched once per group, and against the
        reference's own kernel (BuildGraph::kernel_dynamic, built unmodified)
        launched the same way, on 2,000,000 heavy-tailed protein candidate
        pairs at identity 90, scores compared bit for bit (--pairs N to
        resize, 0 to skip; --pairs-only; --no-plain skips both baselines).
serving (one GPU) queries/s and p50/p99 request latency of the serving engine
        (a resident 2,000,000-protein database, Poisson-arriving requests of
        1-50,000 queries at identity 90, 8 slots) against the same requests
        run one at a time in the plain form, results compared per request
        (--serve-db N to resize, 0 to skip; --serve-only).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

IDENTITY = 95
BANDS = 64
N_SEQS, N_FAMILIES, SEED = 200_000, 20_000, 2
WORKLOAD = "dna_200k_seqs_20k_families_id95_64bands"
DATA = ("synthetic: seeded DNA families (uniform roots 200-3000 nt, GC 0.45, 1-10% subs, "
        "1% indels mean 2), 10 members per family")
# Irreducible integer work of the bit-parallel LCS update per 32 cells (one
# row word, one column): t = V & M; s = V + t + carry; V = s | (V ^ t).
ALIGN_OPS_PER_WORD_STEP = 3
# Logic/shift-pipe work of one band hash in the sketch (per signed position and
# band): the seed xor, four shift+xor pairs, the running min.  Its three
# multiplies issue to the multiply-add pipe alongside and are not counted.
SKETCH_ALU_OPS_PER_HASH = 10
# DRAM bytes (read + write) per unit, from ncu captures of the kernels on the
# 100,000-sequence case of the same generator (profiles/*_dna100k.txt); scaled
# to a full launch by the units it processes (both grow in proportion).
SKETCH_DRAM_BYTES_PER_POSITION = 0.553
SKETCH_TABLE_DRAM_BYTES_PER_POSITION = 0.537  # sketch_rank_kernel, per signed position
ALIGN_DRAM_BYTES_PER_CELL = 4.83e-3  # the align kernels of one step (profiles/align_phase_*)
# The reference's host code clusters about 650 families (6,500 sequences) of
# this generator per second on 16 Grace cores; samples are sized from that.
CPU_FAMILIES_PER_S = 650
CPU_SAMPLE_FAMILIES = 6500
# Batched-vs-plain leg: heavy-tailed protein candidate pairs at identity 90,
# the plain form launched once per group (the reference launches once per band).
PAIRS_N, PAIRS_SEED, PAIRS_IDENTITY, PAIRS_GROUPS = 2_000_000, 3, 90, 64
PAIRS_MAX_STEPS = 5
# Serving leg: a resident database of 2,000,000 proteins (the small-protein
# generator scaled to 100,000 families), 300,000 held-out queries (10 %
# unrelated) in Poisson-arriving requests of log-uniform 1..50,000 queries,
# identity 90; against the same requests run one at a time in the plain form.
SERVE_DB, SERVE_QUERIES, SERVE_FAMILIES, SERVE_SEED, SERVE_IDENTITY = (
    2_000_000, 300_000, 100_000, 4, 90)
SERVE_MAX_BATCH, SERVE_SLOTS, SERVE_LOAD, SERVE_REPLAY = 50_000, 8, 3.0, 10
# Small requests first: requests of at most SERVE_SMALL queries are admitted
# ahead of larger ones, with SERVE_SMALL_SLOTS of the slots kept for them.
SERVE_SMALL, SERVE_SMALL_SLOTS = 256, 2
# Request-size buckets of the latency split (queries per request).
SERVE_SIZE_BUCKETS = ((1, 9), (10, 99), (100, 999), (1000, 9999), (10000, 50000))
# A second serving workload whose queries are close relatives of database
# sequences (families with 0-4 % substitutions and 0.5 % indels of mean 2),
# so that alignment and assignment, not the lookup, dominate.
SERVE_CLOSE_SEED, SERVE_CLOSE_SUBS, SERVE_CLOSE_INDELS = 6, (0.0, 0.04), (0.005, 2.0)
# Streaming leg: a protein database held in host memory (the small-protein
# generator, 12 sequences per family) clustered through 1 GiB of device memory
# for records, 3 rehash rounds at identities 50 and 90; the out-of-HBM
# configuration names 60,000,000 sequences (--stream-seqs 60000000).
STREAM_SEQS, STREAM_PER_FAMILY, STREAM_SEED, STREAM_BANDS = 6_000_000, 12, 5, 3
STREAM_IDENTITIES, STREAM_CHUNK_BYTES = (50, 90), 1 << 30
# The same device step on the small protein configuration: 20,000 proteins
# from 2,000 families (log-normal roots median 300 sigma 0.5, 5-35 % substitutions,
# 2 % indels, seed 1) at identity 90.
PROT_SEQS, PROT_FAMILIES, PROT_SEED, PROT_IDENTITY = 20_000, 2_000, 1, 90
# The command line end to end (FASTA -> packed file -> result file) against the
# reference's own GPU build on the same GPU: both configurations, median of
# REFGPU_REPS runs of each command.
REFGPU_REPS = 3
# The bit-parallel LCS update counted the survey's way: AND, add with carry in,
# carry out, AND-NOT, OR per 32 cells.
ALIGN_OPS_PER_WORD_STEP_5 = 5
# Single-thread row of the CPU baseline: families of the sample (about 10 s of
# the reference's host code on one core).
CPU_SAMPLE_FAMILIES_1T = 500


def log(*a):
    print(*a, file=sys.stderr, flush=True)


def parse():
    p = argparse.ArgumentParser()
    p.add_argument("--gpus", type=int, default=1)
    p.add_argument("--steps", type=int, default=60)
    p.add_argument("--warmup", type=int, default=3)
    p.add_argument("--impl", choices=["ours", "reference"], default="ours")
    p.add_argument("--n-seqs", type=int, default=N_SEQS)
    p.add_argument("--no-cpu-baseline", action="store_true")
    p.add_argument("--ref-families", type=int, default=0,
                   help="families in the CPU samples (default: sized from CPU_FAMILIES_PER_S)")
    p.add_argument("--pairs", type=int, default=PAIRS_N,
                   help="pairs of the batched-vs-plain leg (0 = skip it)")
    p.add_argument("--pairs-only", action="store_true",
                   help="run only the batched-vs-plain leg and print its object")
    p.add_argument("--no-autotune", action="store_true",
                   help="batched leg with the default binning plan")
    p.add_argument("--no-plain", action="store_true",
                   help="skip the plain arm of the batched leg (profiling)")
    p.add_argument("--serve-db", type=int, default=SERVE_DB,
                   help="database sequences of the serving leg (0 = skip it)")
    p.add_argument("--serve-only", action="store_true",
                   help="run only the serving leg and print its object")
    p.add_argument("--stream-seqs", type=int, default=STREAM_SEQS,
                   help="sequences of the streaming leg (0 = skip it)")
    p.add_argument("--stream-only", action="store_true",
                   help="run only the streaming leg and print its object")
    p.add_argument("--stream-check", type=int, default=1,
                   help="1: compare the streamed edges with the resident path's")
    p.add_argument("--stream-chunk-bytes", type=int, default=STREAM_CHUNK_BYTES,
                   help="device bytes for record chunks in the streaming leg")
    p.add_argument("--protein", type=int, default=1,
                   help="1: the device step on the small protein configuration too")
    p.add_argument("--reference-gpu", type=int, default=1,
                   help="1: the command line end to end against the reference's GPU build")
    p.add_argument("--ref-gpu-only", action="store_true",
                   help="run only the command-line comparison and print its object")
    return p.parse_args()


# ---- distributed bookkeeping (replicas: every rank runs the whole workload) --------
def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    pg = None
    if world > 1:
        import torch.distributed as dist
        backend = "nccl" if args.impl == "ours" else "gloo"
        if backend == "nccl":
            import torch
            torch.cuda.set_device(local)
        dist.init_process_group(backend)
        pg = dist
    return world, rank, local, pg


def max_over_ranks(pg, value: float) -> float:
    if pg is None:
        return value
    import torch
    dev = "cuda" if pg.get_backend() == "nccl" else "cpu"
    t = torch.tensor([value], dtype=torch.float64, device=dev)
    pg.all_reduce(t, op=pg.ReduceOp.MAX)
    return float(t.item())


def barrier(pg):
    if pg is not None:
        pg.barrier()


# ---- workload ---------------------------------------------------------------------
def make_database(n_seqs: int, n_families: int, seed: int, workdir: Path):
    import ngia2_gb300 as ng
    from ngia2_gb300 import synth
    t0 = time.time()
    # NGIA_BENCH_CACHE=<dir> keeps the generated workload between runs
    cache = os.environ.get("NGIA_BENCH_CACHE")
    if cache:
        workdir = Path(cache) / f"dna_{n_seqs}_{n_families}_{seed}"
        workdir.mkdir(parents=True, exist_ok=True)
    fasta = workdir / "workload.fa"
    packed = workdir / "workload.packed"
    if not (cache and fasta.exists() and packed.exists()):
        synth.dna_families(n_seqs, n_families, seed).write_fasta(fasta)
        ng.makedb(fasta, packed)
    db = ng.read_packed(packed)
    log(f"workload: {db['n']} sequences, {int(db['lens'].sum())} residues "
        f"({time.time() - t0:.1f} s to generate + makedb)")
    return db, fasta, packed


def signed_positions(lens) -> int:
    """Positions the sketch hashes: L - 7 per record of length L >= 8, one for
    a shorter non-empty record (its whole sequence is the k-mer)."""
    import numpy as np
    lens = np.asarray(lens, dtype=np.int64)
    return int(np.where(lens >= 8, lens - 7, (lens > 0).astype(np.int64)).sum())


class ClockSampler:
    """nvidia-smi clock/throttle samples during the timed region."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.proc = None
        self.gpu = gpu_index
        self.path = Path(tempfile.mkstemp(suffix=".csv")[1])

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.gpu), f"--query-gpu={self.FIELDS}",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None
        # wait (bounded) for the first sample so that sampling covers the timed region
        t0 = time.time()
        while self.proc is not None and time.time() - t0 < 5.0:
            if self.proc.poll() is not None or self.path.stat().st_size > 0:
                break
            time.sleep(0.05)
        return self

    def __exit__(self, *exc):
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.proc.kill()

    def summary(self) -> dict:
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        try:
            for line in self.path.read_text().splitlines():
                f = [x.strip() for x in line.split(",")]
                if len(f) < 9:
                    continue
                try:
                    sm.append(float(f[1]))
                    mx.append(float(f[2]))
                except ValueError:
                    continue
                for k, name in enumerate(names):
                    if f[5 + k].lower().startswith("active"):
                        reasons.add(name)
        except OSError:
            pass
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": max(mx),
                "reasons": sorted(reasons), "samples": len(sm)}


def peaks() -> dict:
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return json.loads(p.read_text())
        except ValueError:
            pass
    return {}


# ---- the reference's CPU implementation --------------------------------------------
class StdoutToStderr:
    """The reference code prints progress on stdout; keep stdout for the one
    JSON line by pointing file descriptor 1 at stderr meanwhile."""

    def __enter__(self):
        sys.stdout.flush()
        self.saved = os.dup(1)
        os.dup2(2, 1)
        return self

    def __exit__(self, *exc):
        import ctypes
        ctypes.CDLL(None).fflush(None)
        os.dup2(self.saved, 1)
        os.close(self.saved)


def reference_step(fasta: Path, workdir: Path) -> tuple[float, dict]:
    """One pass of the reference's own code (host build): makedb + buildGraph."""
    import oracle
    packed = workdir / "ref.packed"
    with StdoutToStderr():
        t0 = time.perf_counter()
        rc = oracle.ref_makedb(fasta, packed)
        t1 = time.perf_counter()
        if rc != 0:
            raise RuntimeError(f"reference makedb failed ({rc})")
        r, _, _ = oracle.ref_build_graph(packed, IDENTITY, BANDS, 1 << 22)
        t2 = time.perf_counter()
    return t2 - t0, {"makedb_s": t1 - t0, "build_graph_s": t2 - t1, "edges": int(len(r))}


def port_step(db) -> tuple[float, dict]:
    """One pass of the C oracle (single thread): sketch, bucket, graph."""
    import numpy as np

    import oracle
    t0 = time.perf_counter()
    sigs = oracle.sketch_all(db["packed"], db["offsets"], db["lens"])
    rep = np.stack([oracle.bucket_band(sigs[b]) for b in range(BANDS)])
    e, _ = oracle.graph_edges(db["packed"], db["offsets"], db["lens"], rep, IDENTITY, BANDS)
    return time.perf_counter() - t0, {"edges": int(len(e))}


def cpu_sample(n_families: int, workdir: Path):
    """A bounded sample of the workload: fewer families, same generator (so the
    per-sequence work distribution is the workload's)."""
    import ngia2_gb300 as ng
    from ngia2_gb300 import synth
    s = synth.dna_families(n_families * (N_SEQS // N_FAMILIES), n_families, SEED + 1000)
    fasta = workdir / "sample.fa"
    s.write_fasta(fasta)
    return fasta, len(s)


def run_cpu_baseline(workdir: Path, steps: int, warmup: int, families: int) -> dict:
    import oracle
    os.environ.setdefault("OMP_NUM_THREADS", str(os.cpu_count() or 1))
    fasta, n = cpu_sample(families, workdir)
    if oracle.ref_available():
        kind, cores = "reference", int(os.environ["OMP_NUM_THREADS"])
        fn = lambda: reference_step(fasta, workdir)  # noqa: E731
    else:
        import ngia2_gb300 as ng
        kind, cores = "port", 1
        ng.makedb(fasta, workdir / "sample.packed")
        db = ng.read_packed(workdir / "sample.packed")
        fn = lambda: port_step(db)  # noqa: E731
    for _ in range(warmup):
        fn()
    times, info = [], {}
    for _ in range(steps):
        t, info = fn()
        times.append(t)
    mean = sum(times) / len(times)
    return {"value": n / mean, "unit": "seqs/s", "cores": cores, "kind": kind,
            "sample": f"{n} sequences ({families} families) of the same generator, "
                      f"identity {IDENTITY}, {BANDS} bands; mean of {steps} passes",
            "seconds_per_pass": mean, "detail": info}


# ---- our arm -----------------------------------------------------------------------
def run_ours(args, world, rank, local, pg):
    import numpy as np
    import torch

    import ngia2_gb300 as ng
    torch.cuda.set_device(local)
    workdir = Path(tempfile.mkdtemp(prefix="ngia_bench_"))
    n_fam = max(1, args.n_seqs // (N_SEQS // N_FAMILIES))
    db, fasta, _ = make_database(args.n_seqs, n_fam, SEED, workdir)
    n = db["n"]
    stream = torch.cuda.Stream()
    ctx = ng.Context(stream.cuda_stream)
    ctx.load(db["packed"], db["offsets"], db["lens"])
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")

    def timed(fn):
        with torch.cuda.stream(stream):
            flush.zero_()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        out = fn()
        b.record(stream)
        b.synchronize()
        return a.elapsed_time(b), out

    step = lambda: ctx.group_align(IDENTITY, BANDS)  # noqa: E731
    for _ in range(args.warmup):
        step()
    barrier(pg)
    torch.cuda.synchronize()
    launches0 = ng.kernel_launches()
    ms, stats = [], []
    with ClockSampler(local) as clk:
        for _ in range(args.steps):
            t, (m, st) = timed(step)
            ms.append(t)
            stats.append(st)
    launches = ng.kernel_launches() - launches0
    torch.cuda.synchronize()
    barrier(pg)
    mean_ms = sum(ms) / len(ms)
    mean_ms_max = max_over_ranks(pg, mean_ms)
    st = stats[-1]
    band_cells = st["aligned_cells"]  # the band cells of every distinct pair
    cells = st["computed_cells"]      # the cells the aligners actually updated
    align_ms = statistics.mean(s["ms_align"] for s in stats)

    # e2e through the C ABI on pinned host buffers
    def pinned(a):
        t = torch.empty(a.nbytes, dtype=torch.uint8, pin_memory=True)
        v = t.numpy().view(a.dtype)
        v[:] = a.reshape(-1)
        return t, v
    _, h_packed = pinned(np.ascontiguousarray(db["packed"]))
    _, h_offs = pinned(np.ascontiguousarray(db["offsets"]))
    _, h_lens = pinned(np.ascontiguousarray(db["lens"]))
    edge_cap = max(1, int(st["unique_pairs"]))
    t_edges = torch.empty(edge_cap * ng.EDGE_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
    h_edges = t_edges.numpy().view(ng.EDGE_DTYPE)
    e2e_step = lambda: ctx.run_host(h_packed, h_offs, h_lens, IDENTITY, BANDS, h_edges)  # noqa
    for _ in range(max(1, args.warmup)):
        e2e_step()
    e2e_ms, e2e_st = [], []
    m_e2e = 0
    for _ in range(args.steps):
        t, (m_e2e, st_e2e) = timed(e2e_step)
        e2e_ms.append(t)
        e2e_st.append(st_e2e)
    e2e_mean = max_over_ranks(pg, sum(e2e_ms) / len(e2e_ms))
    h2d = h_packed.nbytes + h_offs.nbytes + h_lens.nbytes
    d2h = m_e2e * ng.EDGE_DTYPE.itemsize + 8

    if rank != 0:
        ctx.close()
        return None
    int_peak = ng.int32_peak(stream.cuda_stream)
    sketch_ms = statistics.mean(s["ms_sketch"] for s in stats)
    positions = signed_positions(db["lens"])
    hbm = peaks().get("hbm_gbs")
    table_active = ctx.sketch_table_active()

    def roof(kernel, ops, ms, units, unit_name, bytes_per_unit, algo_bytes, launches_):
        achieved = ops / (ms * 1e-3)
        return {"bound": "int32_alu", "kernel": kernel, "achieved": achieved / 1e12,
                "peak": int_peak / 1e12, "unit": "Tops/s (32-bit lane ops)",
                "frac": achieved / int_peak, "peak_source":
                "measured: ngia_int32_peak (lop3 chains on all SMs, the logic/shift pipe)",
                "units": {unit_name: units}, "launches": launches_, "ms": ms,
                "traffic": bytes_per_unit * units / launches_ if bytes_per_unit else None,
                "algorithmic_bytes": algo_bytes / launches_,
                "hbm_frac_of_measured": (algo_bytes / (ms * 1e-3) / (hbm * 1e9)) if hbm else None}

    # the sketch: 64 hashed bands per position (logic-pipe bound), or on a
    # four-letter database the rank walk over the 8-mer orders
    sketch_bytes = int(db["lens"].sum()) / 2 + 4 * BANDS * n  # codes read + signatures
    if table_active:
        achieved = sketch_bytes / (sketch_ms * 1e-3)
        # bound by random shared-memory bits, which no measured peak of this
        # line covers: the figures are of HBM for the input read once
        sketch_roof = {
            "bound": "shared_memory", "kernel": "sketch_rank_kernel (+ sketch_table_kernel for records "
            "under the rank walk's minimum span)",
            "achieved": achieved / 1e9, "peak": hbm, "unit": "GB/s",
            "frac": achieved / (hbm * 1e9) if hbm else None,
            "peak_source": "measured: MEASURED_PEAKS hbm_gbs",
            "units": {"signed_positions": positions}, "launches": 2, "ms": sketch_ms,
            "traffic": SKETCH_TABLE_DRAM_BYTES_PER_POSITION * positions,
            "algorithmic_bytes": sketch_bytes,
            "note": "frac is of HBM, for the input read once; the walk is bound by "
                    "shared-memory bit tests (78 % of its wavefronts' rate, "
                    "profiles/sketch_rank_kernel_dna100k.txt) and issue",
            "hash_equivalent_tops": positions * BANDS * SKETCH_ALU_OPS_PER_HASH
            / (sketch_ms * 1e-3) / 1e12,
            "table_bands": ng.lib().ngia_sketch_table_bands()}
    else:
        sketch_roof = roof("sketch_kernel<NibbleKmers>",
                           positions * BANDS * SKETCH_ALU_OPS_PER_HASH, sketch_ms, positions,
                           "signed_positions", SKETCH_DRAM_BYTES_PER_POSITION, sketch_bytes, 1)
    rs = {
        "sketch": sketch_roof,
        # the align phase: its concurrent launches, timed as a whole
        "align": align_roof(roof, cells, align_ms, int_peak,
                            st["unique_pairs"] * 12 + int(db["lens"].sum()) / 2),
    }
    rs.update(hbm_rooflines(stats, st, n, hbm))
    dominant = max(rs, key=lambda k: rs[k]["ms"])
    line = {
        "metric": "seqs clustered/s", "value": world * n / (mean_ms_max * 1e-3),
        "unit": "seqs/s", "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": mean_ms_max, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "u32", "data": DATA,
        "config": {"workload": WORKLOAD if n == N_SEQS else
                   f"dna_{n}_seqs_{n_fam}_families_id{IDENTITY}_{BANDS}bands",
                   "n_seqs": n, "families": n_fam, "identity": IDENTITY,
                   "bands": BANDS, "stages": "sketch+bucket+candidates+align+emit",
                   "l2": "flushed before every timed step (256 MiB write)",
                   "parallelism": f"replicas x{world}"},
        "aligned_cells_per_s": cells / (mean_ms_max * 1e-3),
        "align_cells_per_s_kernel": cells / (align_ms * 1e-3),
        "stages_ms": {k: statistics.mean(s[k] for s in stats)
                      for k in ("ms_sketch", "ms_bucket", "ms_pairs", "ms_align", "ms_emit")},
        "work": {"candidate_pairs": st["candidate_pairs"], "unique_pairs": st["unique_pairs"],
                 "band_cells": band_cells, "computed_cells": cells, "edges": st["edges"]},
        "roofline": dict(rs[dominant], name=dominant),
        "rooflines": rs,
        "e2e": {"value": world * n / (e2e_mean * 1e-3), "unit": "seqs/s",
                "ms_per_step": e2e_mean, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                # device stages of the host-buffer path (ms_sketch spans the
                # pipelined upload when load_pipelined)
                "stages_ms": {k: statistics.mean(s[k] for s in e2e_st)
                              for k in ("ms_sketch", "ms_bucket", "ms_pairs", "ms_align",
                                        "ms_emit")},
                "load_pipelined": int(min(s["load_pipelined"] for s in e2e_st))},
        "gpu_launches": launches // max(1, args.steps) * args.steps,
        "clocks": clk.summary(),
        "hbm_peak_gbs": peaks().get("hbm_gbs"),
    }
    ctx.close()
    if world == 1 and args.protein:
        # the same device step on the small protein configuration at identity 90
        line["protein"] = run_protein(args, int_peak, hbm)
    if world == 1 and args.reference_gpu:
        # the command line end to end against the reference's own GPU build
        line["reference_gpu"] = run_reference_gpu(fasta)
    if world == 1 and args.pairs > 0:
        # the batched-vs-plain leg on heavy-tailed protein pairs (one GPU)
        line["pairs"] = run_pairs(args)
    if world == 1 and args.serve_db > 0:
        # the serving leg: continuous batching vs per-request plain runs, on the
        # serving configuration and on queries that are close relatives
        line["serving"] = run_serving(args)
        line["serving_close"] = run_serving(args, close=True)
    if world == 1 and args.stream_seqs > 0:
        # the streaming leg: records in host memory, a bounded device budget
        line["stream"] = run_stream(args)
    if world == 1 and not args.no_cpu_baseline:
        try:
            # about 10 s of the reference's host code on all cores
            fam = args.ref_families or CPU_SAMPLE_FAMILIES
            line["cpu_baseline"] = run_cpu_baseline(workdir, 1, 0, fam)
        except Exception as e:  # reported, never silently dropped
            line["cpu_baseline"] = {"value": None, "error": str(e)[:200]}
        try:
            # the same code on one core, on a smaller sample
            line["cpu_baseline"]["single_thread"] = run_cpu_single_thread(workdir)
        except Exception as e:
            line["cpu_baseline"]["single_thread"] = {"value": None, "error": str(e)[:200]}
    return line


def align_roof(roof, cells, align_ms, int_peak, algo_bytes) -> dict:
    """The align phase against the integer-logic peak, with both op counts per
    32 cells: 3 (the update's irreducible ops) and 5 (each of AND, add with
    carry in, carry out, AND-NOT, OR counted)."""
    r = roof("align phase (align_window_kernel per tier of widths / align_group_kernel / "
             "align_wide_kernel)", cells / 32 * ALIGN_OPS_PER_WORD_STEP, align_ms, cells,
             "computed_cells", ALIGN_DRAM_BYTES_PER_CELL, algo_bytes, 1)
    ops5 = cells / 32 * ALIGN_OPS_PER_WORD_STEP_5
    r["ops_per_word_step"] = ALIGN_OPS_PER_WORD_STEP
    r["frac_5_ops_per_word_step"] = ops5 / (align_ms * 1e-3) / int_peak
    return r


def hbm_rooflines(stats, st, n, hbm) -> dict:
    """Bucketing and emission against the measured HBM bandwidth: bucketing
    reads each band's signatures and writes its rep row (4 + 4 bytes per
    sequence and band, 512 per sequence over 64 bands); emission reads each
    distinct pair and its score (8 + 4 bytes) and writes each edge (12 bytes)."""
    out = {}
    for name, ms_key, algo, kernel in (
            ("bucket", "ms_bucket", 8 * BANDS * n,
             "rs_hist/rs_scatter (segmented radix partition) + rep_resolve_kernel / rep_resolve_far_kernel"),
            ("emit", "ms_emit", 12 * st["unique_pairs"] + 12 * st["edges"],
             "emission (few hits: append_hits_kernel / emit_hits_kernel; else emit_sorted)")):
        ms = statistics.mean(s[ms_key] for s in stats)
        achieved = algo / (ms * 1e-3) if ms > 0 else 0.0
        out[name] = {"bound": "hbm", "kernel": kernel, "achieved": achieved / 1e9,
                     "peak": hbm, "unit": "GB/s",
                     "frac": achieved / (hbm * 1e9) if hbm else None,
                     "peak_source": "measured: MEASURED_PEAKS hbm_gbs", "ms": ms,
                     "algorithmic_bytes": algo, "traffic": None}
    # the partition form's own bytes per sequence and band: per pass a digit
    # count (4) and a scatter (read and write key and value, 16), then the
    # resolve (read key and value, write the rep entry: 12)
    passes = 1 if n <= 1 << 10 else 2 if n <= 1 << 18 else 3 if n <= 1 << 26 else 4
    impl = (20 * passes + 12) * BANDS * n
    b = out["bucket"]
    b["partition_passes"] = passes
    b["implementation_bytes"] = impl
    b["implementation_frac"] = impl / (b["ms"] * 1e-3) / (hbm * 1e9) if hbm and b["ms"] else None
    return out


def run_cpu_single_thread(workdir: Path) -> dict:
    """The reference's host build (makedb + clustering through its command
    line) with one OpenMP thread, on a sample of the workload's generator."""
    import oracle
    cli = oracle.REF / "ngia2_cpu_fma"
    if not cli.exists():
        return {"value": None, "error": "reference host build missing"}
    fasta, n = cpu_sample(CPU_SAMPLE_FAMILIES_1T, workdir)
    env = dict(os.environ, OMP_NUM_THREADS="1")
    t0 = time.perf_counter()
    for cmd in (["-m", "makedb", "-f", fasta, "-p", workdir / "st.packed"],
                ["-m", "clustering", "-p", workdir / "st.packed", "-r", workdir / "st.txt",
                 "-i", str(IDENTITY), "-b", str(BANDS)]):
        subprocess.run([str(cli), *map(str, cmd)], check=True, capture_output=True, env=env,
                       timeout=600)
    dt = time.perf_counter() - t0
    return {"value": n / dt, "unit": "seqs/s", "cores": 1, "kind": "reference",
            "sample": f"{n} sequences ({CPU_SAMPLE_FAMILIES_1T} families) of the same generator, "
                      f"identity {IDENTITY}, {BANDS} bands; makedb + clustering (align, "
                      "Leiden, result file) through the reference's command line",
            "seconds": dt}


def run_protein(args, int_peak, hbm) -> dict:
    """The device step (sketch, bucket, candidates, align, emit) on the small
    protein configuration at identity 90, database resident, L2 flushed before
    every step."""
    import torch

    import ngia2_gb300 as ng
    from ngia2_gb300 import synth
    workdir = Path(tempfile.mkdtemp(prefix="ngia_prot_"))
    fa, packed = workdir / "prot.fa", workdir / "prot.packed"
    synth.protein_families(PROT_SEQS, PROT_FAMILIES, PROT_SEED).write_fasta(fa)
    ng.makedb(fa, packed)
    db = ng.read_packed(packed)
    n = db["n"]
    stream = torch.cuda.Stream()
    ctx = ng.Context(stream.cuda_stream)
    ctx.load(db["packed"], db["offsets"], db["lens"])
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")

    def timed():
        with torch.cuda.stream(stream):
            flush.zero_()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        out = ctx.group_align(PROT_IDENTITY, BANDS)
        b.record(stream)
        b.synchronize()
        return a.elapsed_time(b), out

    for _ in range(max(3, args.warmup)):
        timed()
    ms, stats = [], []
    for _ in range(args.steps):
        t, (_, st) = timed()
        ms.append(t)
        stats.append(st)
    ctx.close()
    st = stats[-1]
    mean_ms = statistics.mean(ms)
    align_ms = statistics.mean(s["ms_align"] for s in stats)
    sketch_ms = statistics.mean(s["ms_sketch"] for s in stats)
    positions = signed_positions(db["lens"])
    cells = st["computed_cells"]

    def roof(kernel, ops, ms_, units, unit_name, bytes_per_unit, algo_bytes, launches_):
        achieved = ops / (ms_ * 1e-3)
        return {"bound": "int32_alu", "kernel": kernel, "achieved": achieved / 1e12,
                "peak": int_peak / 1e12, "unit": "Tops/s (32-bit lane ops)",
                "frac": achieved / int_peak, "units": {unit_name: units}, "ms": ms_,
                "traffic": None, "algorithmic_bytes": algo_bytes}
    rs = {"sketch": roof("sketch_kernel<NibbleKmers>", positions * BANDS * SKETCH_ALU_OPS_PER_HASH,
                         sketch_ms, positions, "signed_positions", None,
                         int(db["lens"].sum()) / 2 + 4 * BANDS * n, 1),
          "align": align_roof(roof, cells, align_ms, int_peak,
                              st["unique_pairs"] * 12 + int(db["lens"].sum()) / 2)}
    rs.update(hbm_rooflines(stats, st, n, hbm))
    return {"workload": f"protein_{n}_seqs_{PROT_FAMILIES}_families_id{PROT_IDENTITY}_{BANDS}bands",
            "data": "synthetic: protein families (log-normal roots median 300 sigma 0.5 clipped "
                    "50-1500, background amino-acid frequencies, 5-35% substitutions, 2% indels "
                    "mean 3), shuffled, seed 1",
            "metric": "seqs clustered/s", "value": n / (mean_ms * 1e-3), "unit": "seqs/s",
            "ms_per_step": mean_ms, "steps": args.steps,
            "stages_ms": {k: statistics.mean(s[k] for s in stats)
                          for k in ("ms_sketch", "ms_bucket", "ms_pairs", "ms_align", "ms_emit")},
            "work": {"candidate_pairs": st["candidate_pairs"], "unique_pairs": st["unique_pairs"],
                     "band_cells": st["aligned_cells"], "computed_cells": cells,
                     "edges": st["edges"]},
            "rooflines": rs}


def _timed_cli(cmd) -> tuple[float, str]:
    t0 = time.perf_counter()
    r = subprocess.run([str(c) for c in cmd], capture_output=True, text=True, timeout=1800)
    dt = time.perf_counter() - t0
    if r.returncode != 0:
        raise RuntimeError(f"{cmd[0]} {cmd[1:3]} failed ({r.returncode}): {r.stdout[-400:]}")
    return dt, r.stdout


def _ref_timer(out: str, tag: str):
    """Seconds of the reference's Timer line that follows `tag`."""
    import re
    m = re.search(re.escape(tag) + r"\s*Consuming:\s*(\d+) h\s*(\d+) m\s*(\d+) s\s*(\d+) ms"
                  r"\s*(\d+) us", out)
    if not m:
        return None
    h, mi, sec, ms, us = map(int, m.groups())
    return h * 3600 + mi * 60 + sec + ms / 1e3 + us / 1e6


def run_reference_gpu(dna_fasta: Path) -> dict:
    """FASTA -> packed file -> result file through the command line, this
    build against the reference's own GPU build (its src/main.cu built
    unmodified by nvcc for this GPU), on the same GPU one process at a time:
    makedb then -m clustering (the drop-in flow, two processes each), and this
    build's one-process makedb+clustering.  Median wall time of REFGPU_REPS
    runs per command; packed and result files compared byte for byte."""
    import hashlib

    import ngia2_gb300 as ng
    import oracle
    from ngia2_gb300 import synth
    ref = oracle.ref_gpu_cli()
    if not ref.exists():
        return {"unavailable": "the reference GPU build (oracle/build.sh) is missing"}
    sha = lambda p: hashlib.sha256(Path(p).read_bytes()).hexdigest()  # noqa: E731
    workdir = Path(tempfile.mkdtemp(prefix="ngia_refgpu_"))
    prot_fa = workdir / "prot.fa"
    synth.protein_families(PROT_SEQS, PROT_FAMILIES, PROT_SEED).write_fasta(prot_fa)
    configs = [("protein_20k_seqs_2k_families_id90", prot_fa, PROT_IDENTITY, PROT_SEQS),
               (WORKLOAD, dna_fasta, IDENTITY, N_SEQS)]
    out = {"gpu": "same GPU, one process at a time",
           "reference": "src/main.cu built unmodified: nvcc -O3 -Xcompiler -fopenmp "
                        "-gencode arch=compute_103,code=sm_103 (oracle/build.sh)",
           "reps": REFGPU_REPS, "configs": {}}
    for name, fa, identity, n in configs:
        d = workdir / name
        d.mkdir()
        t = {k: [] for k in ("ref_makedb", "ref_clustering", "ours_makedb", "ours_clustering",
                             "ours_one_process")}
        ref_align = []
        for _ in range(REFGPU_REPS):
            dt, _ = _timed_cli([ref, "-m", "makedb", "-f", fa, "-p", d / "ref.packed"])
            t["ref_makedb"].append(dt)
            dt, o = _timed_cli([ref, "-m", "clustering", "-p", d / "ref.packed", "-r",
                                d / "ref.txt", "-i", identity, "-b", BANDS])
            t["ref_clustering"].append(dt)
            ref_align.append(_ref_timer(o, f"[align {BANDS} bands]"))
            dt, _ = _timed_cli([ng.CLI_PATH, "-m", "makedb", "-f", fa, "-p", d / "ours.packed"])
            t["ours_makedb"].append(dt)
            dt, _ = _timed_cli([ng.CLI_PATH, "-m", "clustering", "-p", d / "ours.packed", "-r",
                                d / "ours.txt", "-i", identity, "-b", BANDS])
            t["ours_clustering"].append(dt)
            dt, _ = _timed_cli([ng.CLI_PATH, "-m", "makedb+clustering", "-f", fa, "-p",
                                d / "one.packed", "-r", d / "one.txt", "-i", identity,
                                "-b", BANDS])
            t["ours_one_process"].append(dt)
        med = {k: statistics.median(v) for k, v in t.items()}
        ref_total = med["ref_makedb"] + med["ref_clustering"]
        ours_total = med["ours_makedb"] + med["ours_clustering"]
        ref_packed = sha(d / "ref.packed")
        out["configs"][name] = {
            "sequences": n, "identity": identity, "bands": BANDS,
            "seconds_median": med,
            "ref_align_seconds_median": statistics.median(a for a in ref_align if a is not None)
            if any(a is not None for a in ref_align) else None,
            "reference_seqs_per_s": n / ref_total,
            "ours_seqs_per_s": n / ours_total,
            "ours_one_process_seqs_per_s": n / med["ours_one_process"],
            "e2e_ratio": ref_total / ours_total,
            "e2e_ratio_one_process": ref_total / med["ours_one_process"],
            "packed_identical": sha(d / "ours.packed") == ref_packed
            and sha(d / "one.packed") == ref_packed,
            "result_identical": sha(d / "ours.txt") == sha(d / "ref.txt")
            and sha(d / "one.txt") == sha(d / "ref.txt"),
        }
    return out


def reference_sample_families(steps: int, warmup: int) -> int:
    """Families per pass of the reference arm: warm-up + timed passes take
    about two minutes of the reference's host code."""
    per_pass_s = 120.0 / max(1, steps + warmup)
    return int(min(CPU_SAMPLE_FAMILIES, max(50, per_pass_s * CPU_FAMILIES_PER_S)))


def run_reference(args, world, rank):
    if rank != 0:
        return None
    workdir = Path(tempfile.mkdtemp(prefix="ngia_ref_"))
    fam = args.ref_families or reference_sample_families(args.steps, args.warmup)
    base = run_cpu_baseline(workdir, args.steps, args.warmup, fam)
    return {
        "metric": "seqs clustered/s", "value": base["value"], "unit": "seqs/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": base["seconds_per_pass"] * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u32", "data": DATA,
        "config": {"workload": WORKLOAD, "identity": IDENTITY, "bands": BANDS,
                   "stages": "makedb (pack+sketch+group) + buildGraph (candidates+align+emit)",
                   "sample": base["sample"]},
        "impl": "reference",
        "cpu_baseline": {k: base[k] for k in ("value", "unit", "cores", "kind", "sample")},
        "e2e": {"value": base["value"], "unit": "seqs/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
        "detail": base.get("detail"),
    }


# ---- batched vs plain on heavy-tailed protein pairs ---------------------------------
def make_pairs(n_pairs: int, workdir: Path):
    """The pair workload as a packed database (through makedb, so the index
    order is the reference's) plus its (rep, tar) pairs."""
    import numpy as np

    import ngia2_gb300 as ng
    from ngia2_gb300 import synth
    t0 = time.time()
    cache = os.environ.get("NGIA_BENCH_CACHE")
    if cache:
        workdir = Path(cache) / f"pairs_{n_pairs}_{PAIRS_SEED}"
        workdir.mkdir(parents=True, exist_ok=True)
    fasta, packed, pfile = workdir / "pairs.fa", workdir / "pairs.packed", workdir / "pairs.npy"
    if not (cache and packed.exists() and pfile.exists()):
        ps = synth.protein_pairs(n_pairs, seed=PAIRS_SEED)
        ps.seqs.write_fasta(fasta)  # already in index order (length descending)
        ng.makedb(fasta, packed)
        np.save(pfile, ps.pairs)
    db = ng.read_packed(packed)
    pairs = np.load(pfile)
    log(f"pairs workload: {len(pairs)} pairs over {db['n']} sequences, "
        f"{int(db['lens'].sum())} residues ({time.time() - t0:.1f} s)")
    return db, pairs


def run_reference_kernel(db, pairs, workdir: Path, want) -> dict:
    """The reference's own alignment kernel (BuildGraph::kernel_dynamic, built
    unmodified by oracle/build.sh) on the same pairs, one launch per group of
    1/PAIRS_GROUPS of them with a synchronisation after each, as the reference
    launches one kernel per band; kernel time from CUDA events in the
    harness, scores compared with the batched round's."""
    import numpy as np

    import oracle
    exe = oracle.ref_gpu_align()
    if not exe.exists():
        return {"ms": None, "error": "reference GPU build missing (oracle/build.sh)"}
    jobs = np.zeros((len(pairs), 3), np.uint32)
    jobs[:, :2] = pairs
    files = {k: workdir / f"ref_{k}.bin" for k in ("packed", "offs", "jobs", "out")}
    np.ascontiguousarray(db["packed"], np.uint32).tofile(files["packed"])
    np.ascontiguousarray(db["offsets"], np.uint64).tofile(files["offs"])
    jobs.tofile(files["jobs"])
    r = subprocess.run([str(exe), str(files["packed"]), str(files["offs"]), str(files["jobs"]),
                        str(PAIRS_IDENTITY), str(files["out"]), str(PAIRS_GROUPS)],
                       capture_output=True, text=True, timeout=1200)
    if r.returncode != 0:
        return {"ms": None, "error": (r.stdout + r.stderr)[-300:]}
    out = json.loads(r.stdout.strip().splitlines()[-1])
    scores = np.fromfile(files["out"], np.uint32).reshape(-1, 3)[:, 2]
    return {"kernel": "BuildGraph::kernel_dynamic (src/buildGraph.hpp:192-253), built "
                      "unmodified, one thread per pair", "ms": out["kernel_ms"],
            "launches": out["groups"], "scores_identical": bool(np.array_equal(scores, want))}


def run_pairs(args) -> dict:
    """Aligned cells/s of the batched aligner (width classes, persistent
    per-class launches) against the plain form (one thread per pair in job
    order, one launch per group of pairs, as the reference launches one
    kernel per band), on the same pairs, with bit-identical scores."""
    import numpy as np
    import torch

    import ngia2_gb300 as ng
    workdir = Path(tempfile.mkdtemp(prefix="ngia_pairs_"))
    db, pairs = make_pairs(args.pairs, workdir)
    m = len(pairs)
    stream = torch.cuda.Stream()
    ctx = ng.Context(stream.cuda_stream)
    ctx.load(db["packed"], db["offsets"], db["lens"])
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()  # noqa
    d_pairs = dev(pairs)
    d_scores = torch.zeros(m, dtype=torch.int32, device="cuda")
    jobs = np.zeros((m, 3), np.uint32)
    jobs[:, :2] = pairs
    d_jobs0 = dev(jobs)
    d_jobs = d_jobs0.clone()
    d_packed, d_offs = dev(db["packed"]), dev(db["offsets"].astype(np.uint64))
    flush = torch.empty(256 << 20, dtype=torch.uint8, device="cuda")
    groups = PAIRS_GROUPS
    bounds = [m * g // groups for g in range(groups + 1)]

    def batched():
        return ctx.align_pairs_device(d_pairs.data_ptr(), m, PAIRS_IDENTITY,
                                      d_scores.data_ptr())

    def plain():
        for g in range(groups):  # one launch per group, synchronised like the reference's
            a, b = bounds[g], bounds[g + 1]
            ng.align_pairs(d_packed.data_ptr(), d_offs.data_ptr(), d_jobs.data_ptr() + 12 * a,
                           b - a, PAIRS_IDENTITY, stream.cuda_stream)
            stream.synchronize()

    def timed(fn):
        with torch.cuda.stream(stream):
            flush.zero_()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        out = fn()
        e1.record(stream)
        e1.synchronize()
        return e0.elapsed_time(e1), out

    steps = max(1, min(args.steps, PAIRS_MAX_STEPS))
    warm = max(1, min(args.warmup, 3))
    # the default binning plan, then the one the autotuner picks on this round
    # (a round's time hangs on its few longest pairs, so a sample misleads)
    default_plan = ctx.plan()
    for _ in range(warm):
        batched()
    t_default = min(timed(batched)[0] for _ in range(steps))
    sample = m
    t0 = time.time()
    plan = default_plan
    if not args.no_autotune:
        plan, _ = ctx.autotune(d_pairs.data_ptr(), sample, PAIRS_IDENTITY, 3)
    tune_s = time.time() - t0
    for _ in range(warm):
        batched()
    tb, st = [], None
    for _ in range(steps):
        t, st = timed(batched)
        tb.append(t)
    tp = []
    if not args.no_plain:
        plain()  # warm-up
        for _ in range(min(steps, 3)):
            t, _ = timed(plain)
            tp.append(t)
    torch.cuda.synchronize()
    got = d_scores.cpu().numpy().view(np.uint32)
    ref = d_jobs.cpu().numpy().view(np.uint32).reshape(-1, 3)[:, 2]
    ref_kernel = None if args.no_plain else run_reference_kernel(db, pairs, workdir, got)
    cells = st["aligned_cells"]
    ms_b = statistics.mean(tb)
    ms_p = statistics.mean(tp) if tp else None
    int_peak = ng.int32_peak(stream.cuda_stream)
    ops = st["computed_cells"] / 32 * ALIGN_OPS_PER_WORD_STEP
    ctx.close()
    return {
        "workload": f"protein_pairs_{m}_heavy_tailed_id{PAIRS_IDENTITY}",
        "data": "synthetic: protein families of 5 (roots 80% log-normal median 250 sigma 0.5, "
                "19% uniform 1k-5k, 1% uniform 5k-35k; members 1-50% subs, 1% indels), "
                "half the pairs within a family, half unrelated neighbours in length order",
        "metric": "aligned cells/s", "unit": "cells/s",
        "note": "band cells of all the pairs, settled early or by the seed filter included",
        "band_cells": cells, "computed_cells": st["computed_cells"],
        "batched": {"value": cells / (ms_b * 1e-3), "ms": ms_b, "steps": steps,
                    "computed_cells_per_s": st["computed_cells"] / (ms_b * 1e-3),
                    "cuda_graph": True, "plan": plan, "autotune_s": tune_s,
                    "autotune_sample_pairs": sample,
                    "ms_default_plan": t_default, "default_plan": default_plan},
        "plain": {"value": cells / (ms_p * 1e-3) if ms_p else None, "ms": ms_p,
                  "launches": groups, "steps": len(tp)},
        "batched_over_plain": ms_p / ms_b if ms_p else None,
        "reference_kernel": ref_kernel,
        "batched_over_reference_kernel": (ref_kernel["ms"] / ms_b
                                          if ref_kernel and ref_kernel.get("ms") else None),
        "roofline": {"bound": "int32_alu", "kernel": "batched round (all width classes)",
                     "achieved": ops / (ms_b * 1e-3) / 1e12, "peak": int_peak / 1e12,
                     "unit": "Tops/s (32-bit lane ops)",
                     "frac": ops / (ms_b * 1e-3) / int_peak,
                     "units": {"computed_cells": st["computed_cells"]}},
        "scores_identical": bool(np.array_equal(got, ref)) if tp else None,
        "hits": int((got > 0).sum()),
    }


# ---- streaming: a database in host memory through a bounded device budget ------------
def make_stream(n: int, workdir: Path):
    import numpy as np

    from ngia2_gb300 import synth
    t0 = time.time()
    cache = os.environ.get("NGIA_BENCH_CACHE")
    d = Path(cache) / f"stream_{n}_{STREAM_SEED}" if cache else workdir
    d.mkdir(parents=True, exist_ok=True)
    files = [d / f"{k}.npy" for k in ("packed", "offs", "lens")]
    if cache and all(f.exists() for f in files):
        packed, offs, lens = (np.load(f) for f in files)
    else:
        packed, offs, lens = synth.packed_proteins(n, max(1, n // STREAM_PER_FAMILY),
                                                   seed=STREAM_SEED)
        if cache:
            for f, a in zip(files, (packed, offs, lens)):
                np.save(f, a)
    log(f"streaming workload: {len(lens)} sequences, {int(lens.sum())} residues, "
        f"{packed.nbytes / 1e9:.2f} GB packed ({time.time() - t0:.1f} s)")
    return packed, offs, lens


def run_stream(args) -> dict:
    """End-to-end seqs/s of the streamed graph build (sketch, bucket, candidates,
    align, emit) with the records in host memory and STREAM_CHUNK_BYTES of device
    memory for them; per stage the host-to-device GB/s; the edges compared with
    the resident path's when --stream-check (and the records fit)."""
    import numpy as np

    import ngia2_gb300 as ng
    workdir = Path(tempfile.mkdtemp(prefix="ngia_stream_"))
    packed, offs, lens = make_stream(args.stream_seqs, workdir)
    n = len(lens)
    # the records in page-locked host memory (set up before timing, as an
    # application holding its database for streaming would), so that chunks
    # go to the device straight from it
    import torch
    t_pin = torch.empty(packed.nbytes, dtype=torch.uint8, pin_memory=True)
    pinned = t_pin.numpy().view(packed.dtype)
    pinned[:] = packed
    packed = pinned
    runs = {}
    k = min(n, 1000)  # warm-up on the first records
    k_words = int(offs[k - 1]) + 1 + 4 * ((int(lens[k - 1]) + 31) // 32)
    budget = args.stream_chunk_bytes
    clk = ClockSampler(torch.cuda.current_device())
    for identity in STREAM_IDENTITIES:
        ng.stream_graph(packed[:k_words], offs[:k], lens[:k], identity, STREAM_BANDS, budget)
        with clk:
            edges, st = ng.stream_graph(packed, offs, lens, identity, STREAM_BANDS, budget,
                                        cap=n * STREAM_BANDS)
        gbs = lambda b, ms: b / (ms * 1e-3) / 1e9 if ms > 0 else None  # noqa: E731
        run = {"value": n / (st["ms_total"] * 1e-3), "unit": "seqs/s", "edges": int(len(edges)),
               "chunks": st["chunks"], "chunk_loads": st["chunk_loads"],
               "stages_ms": {k: st[k] for k in ("ms_sketch", "ms_bucket", "ms_pairs",
                                                "ms_align", "ms_emit", "ms_total")},
               "h2d_gbs": {"sketch": gbs(st["bytes_h2d_sketch"], st["ms_sketch"]),
                           "align": gbs(st["bytes_h2d_align"], st["ms_align"])},
               "h2d_bytes": {"sketch": st["bytes_h2d_sketch"], "align": st["bytes_h2d_align"]},
               "unique_pairs": st["unique_pairs"], "computed_cells": st["computed_cells"],
               "clocks": clk.summary()}
        if args.stream_check:
            with ng.Context() as ctx:
                ctx.load(packed, offs, lens)
                m, _ = ctx.group_align(identity, STREAM_BANDS)
                res = ctx.edges(m)
            run["edges_identical_to_resident"] = bool(
                len(res) == len(edges) and np.array_equal(res["rep"], edges["rep"])
                and np.array_equal(res["tar"], edges["tar"])
                and np.array_equal(res["weight"], edges["weight"]))
        runs[f"id{identity}"] = run
    return {
        "workload": f"stream_{n}_proteins_{STREAM_BANDS}bands",
        "data": "synthetic: small-protein generator (log-normal roots median 300 sigma 0.5, "
                f"5-35% subs, 2% indels), {STREAM_PER_FAMILY} sequences per family, "
                "packed on the device",
        "metric": "seqs/s end to end", "unit": "seqs/s", "sequences": n,
        "packed_bytes": int(packed.nbytes), "device_bytes_for_records": budget,
        "host_records": "page-locked (allocated pinned before timing)",
        "runs": runs,
    }


# ---- serving: continuous batching vs per-request plain runs ---------------------------
def make_serving(n_db: int, workdir: Path, close: bool = False):
    """Database (packed through makedb) and query records of the serving leg;
    close: the close-relatives workload."""
    import ngia2_gb300 as ng
    from ngia2_gb300 import synth
    t0 = time.time()
    scale = n_db / SERVE_DB
    n_q = max(1000, int(SERVE_QUERIES * scale))
    n_fam = max(100, int(SERVE_FAMILIES * scale))
    seed = SERVE_CLOSE_SEED if close else SERVE_SEED
    cache = os.environ.get("NGIA_BENCH_CACHE")
    if cache:
        workdir = Path(cache) / f"serve_{n_db}_{seed}"
        workdir.mkdir(parents=True, exist_ok=True)
    dbp, qp = workdir / "db.packed", workdir / "queries.packed"
    if not (cache and dbp.exists() and qp.exists()):
        kw = {"subs": SERVE_CLOSE_SUBS, "indels": SERVE_CLOSE_INDELS} if close else {}
        db, q = synth.serving_set(n_db, n_q, n_fam, seed=seed, **kw)
        db.write_fasta(workdir / "db.fa")
        q.write_fasta(workdir / "queries.fa")
        ng.makedb(workdir / "db.fa", dbp)
        ng.makedb(workdir / "queries.fa", qp)
    db, q = ng.read_packed(dbp), ng.read_packed(qp)
    log(f"serving workload: {db['n']} database sequences, {q['n']} queries "
        f"({time.time() - t0:.1f} s)")
    return db, q


def serving_requests(q, seed: int = SERVE_SEED):
    """Requests of log-uniform 1..SERVE_MAX_BATCH queries, in a random order
    of the queries: (packed words, local offsets, lengths) each."""
    import numpy as np
    rng = np.random.default_rng(seed + 7)
    n = q["n"]
    order = rng.permutation(n)
    words = 1 + 4 * ((q["lens"].astype(np.int64) + 31) // 32)
    reqs, k = [], 0
    while k < n:
        s = int(min(n - k, max(1, np.floor(np.exp(rng.uniform(0, np.log(SERVE_MAX_BATCH)))))))
        idx = order[k:k + s]
        w = words[idx]
        run = np.concatenate([[0], np.cumsum(w)[:-1]])
        owner = np.repeat(np.arange(s), w)
        gather = q["offsets"][idx].astype(np.int64)[owner] + (np.arange(int(w.sum())) - run[owner])
        reqs.append((np.ascontiguousarray(q["packed"][gather], np.uint32),
                     run.astype(np.uint64), np.ascontiguousarray(q["lens"][idx], np.uint32)))
        k += s
    return reqs


def latency_split(sizes, lat_ms) -> dict:
    """p50/p99 latency (ms) per request-size bucket."""
    import numpy as np
    sizes, lat_ms = np.asarray(sizes), np.asarray(lat_ms)
    out = {}
    for lo, hi in SERVE_SIZE_BUCKETS:
        sel = (sizes >= lo) & (sizes <= hi)
        if sel.any():
            out[f"{lo}-{hi}"] = {"requests": int(sel.sum()),
                                 "p50_ms": float(np.percentile(lat_ms[sel], 50)),
                                 "p99_ms": float(np.percentile(lat_ms[sel], 99))}
    return out


def serve_poisson(srv, reqs, rate: float, seed: int):
    """Requests submitted as Poisson arrivals at `rate` per second; returns the
    per-request (results, stats) and the makespan (first submit -> last done)."""
    import threading

    import numpy as np
    rng = np.random.default_rng(seed)
    gaps = rng.exponential(1.0 / rate, size=len(reqs))
    tickets: list = [None] * len(reqs)
    ready = [threading.Event() for _ in reqs]
    results: list = [None] * len(reqs)
    done_at = [0.0] * len(reqs)

    def waiter():
        for k in range(len(reqs)):
            ready[k].wait()
            results[k] = srv.wait(tickets[k], len(reqs[k][2]))
            done_at[k] = time.perf_counter()

    th = threading.Thread(target=waiter)
    th.start()
    t_begin = time.perf_counter()
    t_next = t_begin
    for k, r in enumerate(reqs):
        t_next += gaps[k]
        delay = t_next - time.perf_counter()
        if delay > 0:
            time.sleep(delay)
        tickets[k] = srv.submit(*r)
        ready[k].set()
    th.join()
    return results, max(done_at) - t_begin


def run_serving(args, close: bool = False) -> dict:
    """p50/p99 latency (overall and per request size) and queries/s of the
    serving engine (continuous batching over SERVE_SLOTS slots, Poisson
    arrivals at SERVE_LOAD x the plain form's request rate), in arrival order
    and with small requests first, against the same requests run one at a
    time in the plain form; per-request results compared."""
    import numpy as np
    import torch

    import ngia2_gb300 as ng
    workdir = Path(tempfile.mkdtemp(prefix="ngia_serve_"))
    db, q = make_serving(args.serve_db, workdir, close)
    reqs = serving_requests(q) * SERVE_REPLAY  # the stream, replayed
    sizes = [len(r[2]) for r in reqs]
    stream = torch.cuda.Stream()
    ctx = ng.Context(stream.cuda_stream)
    ctx.load(db["packed"], db["offsets"], db["lens"])
    t0 = time.time()
    ctx.sketch_bucket(BANDS)
    cluster = ctx.fast_cluster(SERVE_IDENTITY)  # the database's clusters (fast mode)
    t_setup = time.time() - t0
    nq = sum(sizes)

    # plain: one request at a time, plain kernel, no overlap
    plain_out, plain_ms = [], []
    with ng.Server(ctx, cluster, SERVE_IDENTITY, plain=True, max_queries=SERVE_MAX_BATCH) as srv:
        srv.wait(srv.submit(*reqs[0]), len(reqs[0][2]))  # warm-up
        t_begin = time.perf_counter()
        for r in reqs:
            out, st = srv.wait(srv.submit(*r), len(r[2]))
            plain_out.append(out)
            plain_ms.append(st["total_ms"])
        plain_s = time.perf_counter() - t_begin
    plain_rate = len(reqs) / plain_s

    runs = {}
    for name, kw in (("arrival_order", {}),
                     ("small_first", {"small_queries": SERVE_SMALL,
                                      "small_slots": SERVE_SMALL_SLOTS})):
        with ng.Server(ctx, cluster, SERVE_IDENTITY, slots=SERVE_SLOTS,
                       max_queries=SERVE_MAX_BATCH, **kw) as srv:
            srv.wait(srv.submit(*reqs[0]), len(reqs[0][2]))  # warm-up
            results, serve_s = serve_poisson(srv, reqs, SERVE_LOAD * plain_rate, SERVE_SEED + 11)
            # capacity: every request submitted at once
            t_begin = time.perf_counter()
            ts = [srv.submit(*r) for r in reqs]
            for t, r in zip(ts, reqs):
                srv.wait(t, len(r[2]))
            burst_s = time.perf_counter() - t_begin
        lat = np.array([res[1]["total_ms"] for res in results])
        runs[name] = {
            "value": nq / serve_s, "slots": SERVE_SLOTS,
            "arrivals": f"Poisson, {SERVE_LOAD} x the plain request rate",
            "p50_ms": float(np.percentile(lat, 50)), "p99_ms": float(np.percentile(lat, 99)),
            "by_request_size": latency_split(sizes, lat),
            "makespan_s": serve_s, "capacity": nq / burst_s,
            "over_plain": plain_s / serve_s,
            "results_identical": all(np.array_equal(a, b[0])
                                     for a, b in zip(plain_out, results)),
            **({"small_queries": SERVE_SMALL, "small_slots": SERVE_SMALL_SLOTS} if kw else {})}
    pl = np.array(plain_ms)
    assigned = int(sum(int((o != ng.NEW_CLUSTER).sum()) for o in plain_out))
    ctx.close()
    best = max(runs, key=lambda k: runs[k]["value"])
    return {
        "workload": f"serving_db{db['n']}_queries{nq}_id{SERVE_IDENTITY}" +
                    ("_close_relatives" if close else ""),
        "data": "synthetic: small-protein generator (log-normal roots median 300 sigma 0.5, " +
                ("0-4% subs, 0.5% indels mean 2" if close else "5-35% subs, 2% indels") +
                f") scaled to {int(SERVE_FAMILIES * args.serve_db / SERVE_DB)} families; "
                "queries held out of the same families plus 10% unrelated; requests "
                "log-uniform 1-50,000 queries",
        "metric": "queries/s (and request latency)", "unit": "queries/s",
        "requests": len(reqs), "queries": nq, "assigned": assigned,
        "assignment_rate": assigned / nq, "replayed": SERVE_REPLAY,
        "setup_s": t_setup,
        "serving": runs[best], "serving_runs": runs,
        "plain": {"value": nq / plain_s, "p50_ms": float(np.percentile(pl, 50)),
                  "p99_ms": float(np.percentile(pl, 99)), "total_s": plain_s,
                  "by_request_size": latency_split(sizes, pl),
                  "form": "one request at a time, one-thread-per-pair kernel"},
        "serving_over_plain": runs[best]["over_plain"],
        "results_identical": all(r["results_identical"] for r in runs.values()),
    }


def main():
    args = parse()
    world, rank, local, pg = dist_setup(args)
    if args.serve_only:
        import torch
        torch.cuda.set_device(local)
        print(json.dumps({"serving": run_serving(args),
                          "serving_close": run_serving(args, close=True)}), flush=True)
        return
    if args.stream_only:
        import torch
        torch.cuda.set_device(local)
        print(json.dumps(run_stream(args)), flush=True)
        return
    if args.pairs_only:
        import torch
        torch.cuda.set_device(local)
        print(json.dumps(run_pairs(args)), flush=True)
        return
    if args.ref_gpu_only:
        _, fasta, _ = make_database(args.n_seqs, max(1, args.n_seqs // (N_SEQS // N_FAMILIES)),
                                    SEED, Path(tempfile.mkdtemp(prefix="ngia_bench_")))
        print(json.dumps(run_reference_gpu(fasta)), flush=True)
        return
    if args.impl == "reference":
        line = run_reference(args, world, rank)
    else:
        line = run_ours(args, world, rank, local, pg)
    if pg is not None:
        pg.destroy_process_group()
    if line is not None and rank == 0:
        print(json.dumps(line), flush=True)


if __name__ == "__main__":
    main()
