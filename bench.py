"""Benchmark of the batched mixed-k max_zeros path on B200 GPUs.

Workload (one step): 10,000 seeded random exponent sets P of Z_7^2 with |P|
uniform in 6..14 (distinct indices), target_distance = 1 (no early exit),
every set's exact max_zeros -- the batched uneven evaluation configuration.
Metric: reference-equivalent codewords/s = sum over the sets of (8^k - 1),
the messages the reference enumerates per set, divided by the step time.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl b200|reference]

N > 1 runs one process per GPU under torch.distributed.run; every rank
evaluates its own seeded batch (weak scaling, no collective on the data path)
and the step time is the maximum over ranks.  `--impl reference` times the
reference algorithm on the host cores (the CPU restatement of kernel.py's
batched enumeration) on a bounded sample of the same workload.
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

import numpy as np

ROOT = Path(__file__).resolve().parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

N_SETS = 10_000
K_LO, K_HI = 6, 14
BASE_SEED = 20260
METRIC = "GF(8) codewords/s, reference-equivalent (8^k-1 messages per code), batched mixed-k"
UNIT = "codewords/s"
WORKLOAD = "batched uneven evaluation: 10,000 seeded random P, |P|~U{6..14}, td=1, exact"
POPC_PER_CODEWORD = 14.0 / 8.0  # histogram walk: 7 bins x 2 words per 8 codewords
# toric_walk_kernel: a carry-save adder over 30 columns' bit rows takes 54 LOP3
# per 32 codewords (the fewest columns it counts: codes of up to 12 rows count
# 36 or 42, so the executed LOP3 are more)
LOP3_PER_CODEWORD_TORIC_WALK = 54.0 / 32.0
# DRAM traffic of one toric_walk_kernel launch (dram__bytes.sum) from an ncu
# capture of 1000 sets of k = 14 (4.75e9 codewords): the walk reads each set's
# tables (112 bytes per row) and keeps everything else on the SM.
TORIC_WALK_DRAM_BYTES = 2.0e6
# toric_prep_kernel: per sweep of 7 codewords, 7 counts on the low 32 columns
# and one of the columns that no coefficient makes zero (the fewest: sweeps over
# all columns count both words)
POPC_PER_CODEWORD_TORIC_PREP = 8.0 / 7.0


# --enumeration: (TG_ENUM_* value, description)
ENUMERATIONS = {
    "auto": (0, "auto: information sets for k >= 2, orbit (projective + torus "
                "normalisation) below"),
    "projective": (1, "projective messages"),
    "orbit": (2, "orbit (projective + torus normalisation)"),
    "infoset": (3, "information sets for every set"),
}


def last_infoset_level(k_max: int) -> int:
    """The last level the information-set walk launches for the toric matrix
    (tg_infoset_last_level): the smallest L with ceil(49 (L + 1) / k) above
    the Griesmer cap of a [49, k] code over GF(8), maximised over k <= k_max."""
    import math

    last = 0
    for k in range(1, k_max + 1):
        cap = max(d for d in range(1, 50)
                  if sum(math.ceil(d / 8 ** i) for i in range(k)) <= 49)
        L = 0
        while math.ceil(49 * (L + 1) / k) < cap + 1:
            L += 1
        last = max(last, min(L, k))
    return last


def takes_toric_walk(k_max: int, enumeration: str) -> bool:
    """Whether an exact batch of the toric matrix goes to toric_prep_kernel and
    toric_walk_kernel (the rule of bind_distance, csrc/abi.cu)."""
    return k_max >= 2 and enumeration in ("auto", "infoset")


def launches_per_step(k_max: int, enumeration: str) -> int:
    """Kernels per step of the general walks: prep_exact, scan_tasks and the
    enumeration walk; with information sets also prep_infoset, order_codes, levels123 (levels 1 to
    3), per level 4..last_infoset_level(k_max) two parts of plan, scan and
    walk each, and finalize_infoset."""
    infoset = enumeration == "infoset" or (enumeration == "auto" and k_max >= 2)
    return 3 + ((4 + 6 * max(0, last_infoset_level(k_max) - 3)) if infoset else 0)


def step_launches(k_max: int, enumeration: str) -> int:
    """Kernels per step of a toric batch: toric_prep_kernel and
    toric_walk_kernel, or the general walks'."""
    return 2 if takes_toric_walk(k_max, enumeration) else launches_per_step(k_max, enumeration)


def roofline(toric: bool, prep_s: float, enum_s: float, infoset_s: float, prep_codewords: int,
             paths: dict, pipes: dict, sm_count: int, mhz: float) -> dict:
    """The dominant kernel of a step against the integer pipe that bounds it:
    of a toric batch the longer of its two kernels, each with the codewords it
    evaluates itself, else the walk over all messages."""
    if not toric:
        kernel, seconds, codewords = "walk_hist_kernel", enum_s, paths["enumeration_codewords"]
        pipe, per, note = "popc", POPC_PER_CODEWORD, "14 POPC per 8-codeword histogram"
    elif infoset_s >= prep_s:
        kernel, seconds = "toric_walk_kernel", infoset_s
        codewords = paths["infoset_codewords"] - prep_codewords
        pipe, per = "lop3", LOP3_PER_CODEWORD_TORIC_WALK
        note = ("54 LOP3 per 32 codewords, the carry-save adder over 30 columns; the kernel "
                "executes more (36 or 42 columns for k <= 12, offsets, the bit rows' build)")
    else:
        kernel, seconds, codewords = "toric_prep_kernel", prep_s, prep_codewords
        pipe, per = "popc", POPC_PER_CODEWORD_TORIC_PREP
        note = ("8 POPC per sweep of 7 codewords over the low 32 columns; the kernel executes "
                "more (both words up to k = 10 and below level 4)")
    clocks = sm_count * mhz * 1e6  # SM clocks a second
    peak = pipes.get(f"{pipe}_per_clk_sm", {"lop3": 64.0, "popc": 16.0}[pipe]) * clocks
    achieved = per * codewords / seconds
    traffic = {"traffic": TORIC_WALK_DRAM_BYTES,
               "traffic_unit": "bytes per launch (ncu, 1000 sets of k = 14, 4.75e9 codewords)"} \
        if kernel == "toric_walk_kernel" else {}
    return {"bound": f"int ({pipe.upper()})", "achieved": achieved / 1e12, "peak": peak / 1e12,
            "unit": f"T{pipe}/s", "frac": achieved / peak, "kernel": kernel,
            "codewords": int(codewords),
            "codewords_per_clk_sm": codewords / seconds / clocks,
            "kernel_share": seconds / (prep_s + enum_s + infoset_s),
            "note": note + f"; peak = measured {pipe.upper()}/clk/SM x SMs x median SM MHz in "
                           "the timed region", **traffic}


L2_FLUSH_BYTES = 256 << 20


def make_workload(rank: int, n: int = N_SETS, k_lo: int = K_LO, k_hi: int = K_HI):
    """Seeded batch of rank `rank` (rank 0 is the headline batch)."""
    rng = np.random.default_rng(BASE_SEED + rank)
    ks = rng.integers(k_lo, k_hi + 1, size=n)
    return [sorted(rng.choice(49, int(k), replace=False).tolist()) for k in ks]


def shard_bounds(n: int, rank: int, world: int) -> tuple[int, int]:
    """Contiguous near-equal shard [lo, hi) of n items for `rank` (used when a
    fixed batch is split across ranks)."""
    q, r = divmod(n, world)
    lo = rank * q + min(rank, r)
    return lo, lo + q + (1 if rank < r else 0)


def stratified_sample(sets, per_k: int) -> dict[int, list[list[int]]]:
    out: dict[int, list[list[int]]] = {}
    for s in sets:
        lst = out.setdefault(len(s), [])
        if len(lst) < per_k:
            lst.append(s)
    return out


def k_histogram(sets) -> dict[int, int]:
    h: dict[int, int] = {}
    for s in sets:
        h[len(s)] = h.get(len(s), 0) + 1
    return h


# ---------------------------------------------------------------------------
# distributed plumbing
# ---------------------------------------------------------------------------

class Dist:
    def __init__(self):
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.rank = int(os.environ.get("RANK", "0"))
        self.local_rank = int(os.environ.get("LOCAL_RANK", "0"))
        self.pg = None

    def init(self, backend: str) -> None:
        if self.world > 1:
            import datetime

            import torch.distributed as dist

            os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
            dist.init_process_group(backend, timeout=datetime.timedelta(seconds=600))
            self.pg = dist

    def barrier(self) -> None:
        if self.pg is not None:
            self.pg.barrier()

    def max(self, x: float, device=None) -> float:
        if self.pg is None:
            return x
        import torch

        t = torch.tensor([x], dtype=torch.float64, device=device)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.MAX)
        return float(t.item())

    def sum(self, x: float, device=None) -> float:
        if self.pg is None:
            return x
        import torch

        t = torch.tensor([x], dtype=torch.float64, device=device)
        self.pg.all_reduce(t, op=self.pg.ReduceOp.SUM)
        return float(t.item())

    def close(self) -> None:
        if self.pg is not None:
            self.pg.destroy_process_group()


# ---------------------------------------------------------------------------
# clocks during the timed region
# ---------------------------------------------------------------------------

class NvmlClockSampler:
    """Samples SM clock, power and clock-event reasons every `period` seconds
    from a thread through NVML (read-only queries)."""

    REASONS = {"hw_slowdown": "nvmlClocksEventReasonHwSlowdown",
               "hw_thermal_slowdown": "nvmlClocksEventReasonHwThermalSlowdown",
               "sw_thermal_slowdown": "nvmlClocksEventReasonSwThermalSlowdown",
               "sw_power_cap": "nvmlClocksEventReasonSwPowerCap"}

    def __init__(self, cuda_index: int, period: float = 0.005):
        import threading

        import pynvml
        import torch

        self.nv = pynvml
        pynvml.nvmlInit()
        handle = None
        try:
            uuid = str(torch.cuda.get_device_properties(cuda_index).uuid)
            handle = pynvml.nvmlDeviceGetHandleByUUID(
                uuid if uuid.startswith("GPU-") else "GPU-" + uuid)
        except Exception:  # noqa: BLE001 - fall back to the index
            handle = pynvml.nvmlDeviceGetHandleByIndex(cuda_index)
        self.h = handle
        self.period = period
        self.rows: list[tuple] = []
        self._stop = threading.Event()
        self._thread = threading.Thread(target=self._run, daemon=True)

    def _run(self) -> None:
        nv = self.nv
        while not self._stop.is_set():
            try:
                self.rows.append((nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM),
                                  nv.nvmlDeviceGetPowerUsage(self.h) / 1000.0,
                                  nv.nvmlDeviceGetCurrentClocksEventReasons(self.h)))
            except Exception:  # noqa: BLE001 - a failed read is skipped
                pass
            self._stop.wait(self.period)

    def start(self) -> None:
        self._thread.start()

    def stop(self) -> dict:
        self._stop.set()
        self._thread.join(timeout=5)
        nv = self.nv
        try:
            smax = nv.nvmlDeviceGetMaxClockInfo(self.h, nv.NVML_CLOCK_SM)
        except Exception:  # noqa: BLE001
            smax = None
        if not self.rows:
            return {"sm_mhz": None, "sm_max_mhz": smax, "reasons": ["no samples"]}
        reasons = set()
        for _, _, mask in self.rows:
            for name, attr in self.REASONS.items():
                if mask & getattr(nv, attr, 0):
                    reasons.add(name)
        return {"sm_mhz": statistics.median(r[0] for r in self.rows), "sm_max_mhz": smax,
                "reasons": sorted(reasons), "samples": len(self.rows),
                "power_w_max": max(r[1] for r in self.rows), "source": "nvml"}


def clock_sampler(cuda_index: int):
    """NVML sampler when available, else nvidia-smi."""
    try:
        return NvmlClockSampler(cuda_index)
    except Exception:  # noqa: BLE001 - no NVML: nvidia-smi
        return ClockSampler(cuda_index)


class ClockSampler:
    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu_index = gpu_index
        self.proc = None
        self.path = None

    def start(self) -> None:
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu_index}", f"--query-gpu={self.QUERY}",
                 "--format=csv,noheader,nounits", "-lms", "20"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        rows = []
        for line in Path(self.path).read_text().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) >= 9:
                rows.append(f)
        os.unlink(self.path)
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}

        def num(x):
            try:
                return float(x)
            except ValueError:
                return None

        sm = [num(r[1]) for r in rows if num(r[1])]
        smax = [num(r[2]) for r in rows if num(r[2])]
        reasons = set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            for name, val in zip(names, r[5:9]):
                if val.lower() in ("active", "yes"):
                    reasons.add(name)
        return {"sm_mhz": statistics.median(sm) if sm else None,
                "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(rows),
                "power_w_max": max((num(r[3]) or 0.0) for r in rows)}


# ---------------------------------------------------------------------------
# CPU baseline (the reference algorithm on the host cores)
# ---------------------------------------------------------------------------

def cpu_reference_rate(sets, prefix: int, per_k: int = 2, threads: int = 0) -> dict:
    """Reference-equivalent codewords/s of the CPU restatement of kernel.py's
    batched enumeration on the workload's k mix, from bounded prefixes of
    `per_k` sets per k (per-message cost grows with k, so the rate is the
    workload-weighted harmonic mean)."""
    from oracle import oracle as orc

    M = orc.eval_matrix()
    threads = threads or os.cpu_count() or 1
    hist = k_histogram(sets)
    sample = stratified_sample(sets, per_k)
    t_msg: dict[int, float] = {}
    total_msgs = 0
    total_s = 0.0
    for k, group in sorted(sample.items()):
        t0 = time.perf_counter()
        msgs, _ = orc.eval_prefix_batch(M, group, prefix, threads=threads)
        dt = time.perf_counter() - t0
        t_msg[k] = dt / max(msgs, 1)
        total_msgs += msgs
        total_s += dt
    work = sum(hist[k] * ((8 ** k) - 1) for k in hist)
    secs = sum(hist[k] * ((8 ** k) - 1) * t_msg[k] for k in hist)
    return {"value": work / secs, "unit": UNIT, "cores": threads, "kind": "port",
            "sample": (f"{per_k} sets per k in {K_LO}..{K_HI}, messages 1..min(8^k-1, {prefix}) "
                       f"each ({total_msgs:.3g} messages, {total_s:.1f} s), rate weighted by the "
                       f"10,000-set k mix"),
            "seconds": total_s}


def run_reference_arm(args, d: Dist) -> None:
    if d.rank != 0:
        return
    sets = make_workload(0, args.n_sets, args.kmin, args.kmax)
    prefix = 1 << 24
    for _ in range(args.warmup):
        cpu_reference_rate(sets, prefix)
    vals = []
    secs = 0.0
    for _ in range(args.steps):
        r = cpu_reference_rate(sets, prefix)
        vals.append(r["value"])
        secs += r["seconds"]
    value = statistics.median(vals)
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT,
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * secs / max(args.steps, 1), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u64 (bit-sliced GF(8))",
        "data": "synthetic (seeded)", "config": {"workload": WORKLOAD, "sample": r["sample"]},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": r["cores"], "kind": "port",
                         "sample": r["sample"]},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


# ---------------------------------------------------------------------------
# Secondary configurations (rank 0, reported beside the headline)
# ---------------------------------------------------------------------------

# Best-known minimum distances of [49, k] codes over GF(8) bundled with the
# reference's evolutionary notebook (used when codetables.de is unreachable).
FALLBACK_BEST_D = {12: 28, 13: 27, 14: 26, 15: 24, 16: 24, 17: 23, 18: 21, 19: 21}


def random_masks(n: int, k_lo: int, k_hi: int, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    keys = rng.random((n, 49))
    ks = rng.integers(k_lo, k_hi + 1, size=n)
    order = np.argsort(keys, axis=1)
    sel = np.arange(49)[None, :] < ks[:, None]
    bits = np.zeros((n, 49), dtype=bool)
    np.put_along_axis(bits, order, sel, axis=1)
    return (bits.astype(np.uint64) << np.arange(49, dtype=np.uint64)).sum(axis=1, dtype=np.uint64)


def bench_canonical(dev: int, n: int = 1_000_000, with_cpu: bool = True) -> dict:
    """Canonical forms of n seeded 49-bit sets (popcount U{5..30}) and device
    dedup of the canonical masks."""
    import torch

    from generalized_toric_gpu_search_b200 import _lib
    from generalized_toric_gpu_search_b200.canonical import CanonicalDedup, CanonicalOracle

    masks = random_masks(n, 5, 30, BASE_SEED + 3)
    co = CanonicalOracle(dev)
    d_in = torch.from_numpy(masks.view(np.int64)).to(f"cuda:{dev}")
    out = torch.empty(n, dtype=torch.int64, device=f"cuda:{dev}")
    s = torch.cuda.current_stream(dev)
    lib = _lib.load()

    def run():
        _lib.check(lib.tg_canonical_masks(co.ctx.handle, d_in.data_ptr(), n, out.data_ptr(),
                                          None, None, s.cuda_stream), "tg_canonical_masks")

    run()
    torch.cuda.synchronize()
    e = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
    dd = CanonicalDedup(dev, capacity=1 << 22)
    dd.insert_device(out[:1024], stream=s)  # loads the hash kernels before the timed insert
    dd.clear(stream=s)
    torch.cuda.synchronize()
    e[0].record(s)
    run()
    e[1].record(s)
    e[2].record(s)
    _, n_new, _ = dd.insert_device(out, stream=s)
    e[3].record(s)
    torch.cuda.synchronize()
    t_canon = e[0].elapsed_time(e[1]) / 1e3
    t_dedup = e[2].elapsed_time(e[3]) / 1e3
    out = {"workload": f"{n:,} seeded 49-bit sets, popcount U{{5..30}}",
           "canonical_sets_per_s": n / t_canon, "canonical_ms": 1e3 * t_canon,
           "dedup_ms": 1e3 * t_dedup, "unique": int(n_new.item())}
    out["reference_gpu"] = canonical_reference_kernel(dev, masks, co, lib)
    if with_cpu:
        out["cpu_baseline"] = canonical_cpu_baseline(masks)
    return out


def _rows_of(masks: np.ndarray) -> list[list[int]]:
    return [[i for i in range(49) if (int(m) >> i) & 1] for m in masks.tolist()]


def canonical_reference_kernel(dev: int, masks: np.ndarray, co, lib, n: int = 200_000) -> dict:
    """The reference canonical kernel (kernel_canon.py:44-129, one warp per
    set, one launch per set size as CanonicalOracle.compute takes (n, k)
    arrays) against this repository's on the same sets: the first n masks of
    popcount <= 16 (the reference key's limit), grouped by popcount."""
    import torch

    from generalized_toric_gpu_search_b200 import _lib
    from generalized_toric_gpu_search_b200.tables import precompute_gl2_perms, rel_table

    ref = _ref_kernels()
    if ref is None:
        return {"unavailable": "oracle/_ref/libref_kernels.so not built"}
    device = torch.device("cuda", dev)
    pc = np.array([bin(int(m)).count("1") for m in masks[: 4 * n].tolist()])
    sel = masks[: 4 * n][pc <= 16][:n]
    rows = _rows_of(sel)
    by_k: dict[int, list] = {}
    for r in rows:
        by_k.setdefault(len(r), []).append(r)
    perms = torch.from_numpy(precompute_gl2_perms()).to(device)
    rel = torch.from_numpy(rel_table()).to(device)
    st = torch.cuda.current_stream(device)
    t_ref = t_ours = 0.0
    for k, group in sorted(by_k.items()):
        d_sets = torch.tensor(group, dtype=torch.int32, device=device)
        m = len(group)
        lo = torch.full((m,), -1, dtype=torch.int64, device=device)
        hi = torch.zeros(m, dtype=torch.int64, device=device)
        om = torch.empty(m, dtype=torch.int64, device=device)
        ol, oh = torch.empty_like(om), torch.empty_like(om)
        for rep_ in range(2):  # the first pass warms both modules
            e = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
            e[0].record(st)
            ref.ref_canon(d_sets.data_ptr(), perms.data_ptr(), rel.data_ptr(), lo.data_ptr(),
                          hi.data_ptr(), m, k, st.cuda_stream)
            e[1].record(st)
            _lib.check(lib.tg_canonical_sets(co.ctx.handle, d_sets.data_ptr(), m, k,
                                             om.data_ptr(), ol.data_ptr(), oh.data_ptr(), None,
                                             st.cuda_stream), "tg_canonical_sets")
            e[2].record(st)
            e[2].synchronize()
        t_ref += e[0].elapsed_time(e[1]) / 1e3
        t_ours += e[1].elapsed_time(e[2]) / 1e3
        if not (torch.equal(lo, ol) and torch.equal(hi, oh)):
            raise SystemExit(f"canonical keys differ from the reference kernel at k = {k}")
    return {"sets": len(rows), "sample": f"first {len(rows):,} masks with popcount <= 16, one "
                                         "launch per popcount",
            "reference_sets_per_s": len(rows) / t_ref, "ours_sets_per_s": len(rows) / t_ours,
            "speedup": t_ref / t_ours, "keys_equal": True}


def _numpy_canonical_chunk(args):
    from oracle import oracle as orc

    k, rows = args
    return len(orc.canonical_forms_numpy(np.array(rows, dtype=np.int32)))


def canonical_cpu_baseline(masks: np.ndarray, n_c: int = 200_000, n_np: int = 8_000) -> dict:
    """CPU baselines of the canonical form on the host's cores: the C
    restatement of kernel_canon.py (OpenMP, every popcount) on the first n_c
    masks, and the numpy restatement of the reference's canonical_forms_batch
    (champion_search_canonical.py:115-140, k <= 10) in a process pool of one
    worker per core on the first n_np masks of popcount <= 10."""
    import multiprocessing as mp

    from oracle import oracle as orc

    cores = os.cpu_count() or 1
    sub = masks[:n_c]
    t0 = time.perf_counter()
    orc.canonical_masks(sub, threads=cores)
    t_c = time.perf_counter() - t0
    pc = np.array([bin(int(m)).count("1") for m in masks[: 4 * n_np].tolist()])
    rows = _rows_of(masks[: 4 * n_np][pc <= 10][:n_np])
    chunks = []
    by_k: dict[int, list] = {}
    for r in rows:
        by_k.setdefault(len(r), []).append(r)
    for k, group in by_k.items():
        step = max(1, len(group) // cores + 1)
        chunks += [(k, group[i:i + step]) for i in range(0, len(group), step)]
    with mp.get_context("spawn").Pool(cores) as pool:
        pool.map(_numpy_canonical_chunk, [(5, [[0, 1, 2, 3, 4]])] * cores)  # start the workers
        t0 = time.perf_counter()
        done = sum(pool.map(_numpy_canonical_chunk, chunks))
        t_np = time.perf_counter() - t0
    return {"value": len(sub) / t_c, "unit": "sets/s", "cores": cores, "kind": "port",
            "sample": f"first {len(sub):,} masks (popcount 5..30), C restatement, OpenMP",
            "numpy_reference_restated": {"value": done / t_np, "unit": "sets/s",
                                         "cores": cores,
                                         "sample": f"first {done:,} masks of popcount <= 10, "
                                                   "canonical_forms_batch restated in numpy, "
                                                   "spawn pool of one process per core"}}


REF_LIB = ROOT / "oracle" / "_ref" / "libref_kernels.so"


def _ref_kernels():
    """The reference's own CUDA kernels, built from its kernel source by
    oracle/build_ref.py and launched with its wrappers' geometry by
    oracle/ref_harness.cu (a baseline here, never the measured product), or
    None when the library was not built."""
    import ctypes

    if not REF_LIB.exists():
        return None
    lib = ctypes.CDLL(str(REF_LIB))
    vp = ctypes.c_void_p
    lib.ref_bp_batch.argtypes = [vp, vp, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                                 ctypes.c_longlong, ctypes.c_ulonglong, vp, vp]
    lib.ref_bp_single.argtypes = [vp, vp, ctypes.c_int, ctypes.c_int, vp, vp]
    lib.ref_canon.argtypes = [vp, vp, vp, vp, vp, ctypes.c_int, ctypes.c_int, vp]
    return lib


def bench_reference_gpu(dev: int, sets, full: int = 1184, ks=(6, 7, 8, 9)) -> dict:
    """The plain GPU form of the reference on this B200:
    eval_min_distance_batch_bp (kernel_cuda_bp.py:146-238), one launch per
    uniform-k group (the only batching its max_zeros_batch offers), and
    eval_min_distance_single_bp (:266-288), one launch per code.  Each is
    timed with CUDA events at k = 6..9 -- the batch kernel on `full` sets per
    launch (8 blocks of 256 threads per SM, full occupancy), the single-set
    kernel on 4 codes per k.  A full launch above k = 9 takes from ~10 s to
    hours, so the time per message at k = 10..14 comes from the least-squares
    line t(k) = a + b k through the measured k (the inner loop is k
    shared-memory lookups per message), applied to the workload's k mix."""
    import torch

    from generalized_toric_gpu_search_b200.tables import build_eval_matrix

    lib = _ref_kernels()
    if lib is None:
        return {"unavailable": "oracle/_ref/libref_kernels.so not built"}
    device = torch.device("cuda", dev)
    d_M = torch.from_numpy(np.ascontiguousarray(build_eval_matrix().astype(np.int32))).to(device)
    st = torch.cuda.current_stream(device)
    by_k: dict[int, list] = {}
    for s_ in sets:
        by_k.setdefault(len(s_), []).append(s_)

    def timed(fn) -> float:
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(st)
        fn()
        e1.record(st)
        e1.synchronize()
        return e0.elapsed_time(e1) / 1e3

    batch_t, single_t = {}, {}
    for k in ks:
        group = by_k[k]
        rows = [group[i % len(group)] for i in range(full)]
        flat = torch.tensor([i for r in rows for i in r], dtype=torch.int32, device=device)
        out = torch.zeros(full, dtype=torch.int32, device=device)
        lib.ref_bp_batch(d_M.data_ptr(), flat.data_ptr(), k, 48, 8, 0, 0, out.data_ptr(),
                         st.cuda_stream)  # warm-up launch
        secs = timed(lambda: lib.ref_bp_batch(d_M.data_ptr(), flat.data_ptr(), k, 48, full, 0, 0,
                                              out.data_ptr(), st.cuda_stream))
        batch_t[k] = secs / (full * float(8 ** k - 1))
        one = torch.zeros(1, dtype=torch.int32, device=device)
        tot = 0.0
        for r in group[:4]:
            d_s = torch.tensor(r, dtype=torch.int32, device=device)
            one.zero_()
            tot += timed(lambda: lib.ref_bp_single(d_M.data_ptr(), d_s.data_ptr(), k, 48,
                                                   one.data_ptr(), st.cuda_stream))
        single_t[k] = tot / (4 * float(8 ** k - 1))
    hist = k_histogram(sets)
    msgs = sum(hist[k] * float(8 ** k - 1) for k in hist)

    def total_seconds(t_by_k):
        kk = np.array(sorted(t_by_k), dtype=np.float64)
        b, a = np.polyfit(kk, np.array([t_by_k[int(k)] for k in kk]), 1)
        per = {k: (t_by_k[k] if k in t_by_k else a + b * k) for k in hist}
        return sum(hist[k] * float(8 ** k - 1) * per[k] for k in hist), per

    batch_s, batch_per = total_seconds(batch_t)
    single_s, single_per = total_seconds(single_t)
    return {"kernel": "reference eval_min_distance_batch_bp / eval_min_distance_single_bp "
                      "(built from kernel_cuda_bp.py's source for sm_100a)",
            "batched_per_k_launch": {"value": msgs / batch_s, "unit": UNIT,
                                     "messages_per_s_measured": {k: 1.0 / t for k, t in
                                                                 batch_t.items()}},
            "one_code_per_launch": {"value": msgs / single_s, "unit": UNIT,
                                    "messages_per_s_measured": {k: 1.0 / t for k, t in
                                                                single_t.items()}},
            "step_seconds_batched": batch_s, "step_seconds_one_per_launch": single_s,
            "sample": f"measured at k = {list(ks)} ({full} sets per batch launch, 4 single-set "
                      f"launches per k); k = {sorted(set(hist) - set(ks))} extrapolated by "
                      "t(k) = a + b k per message"}


def bench_early_exit(dev: int, n: int = 2000) -> dict:
    """n seeded sets of k = 15 against the k = 15 best-known distance."""
    from generalized_toric_gpu_search_b200.distance import DistanceOracleCUDABP
    from generalized_toric_gpu_search_b200.tables import build_eval_matrix

    rng = np.random.default_rng(BASE_SEED + 5)
    sets = [sorted(rng.choice(49, 15, replace=False).tolist()) for _ in range(n)]
    td = FALLBACK_BEST_D[15]
    o = DistanceOracleCUDABP(dev, build_eval_matrix())
    o.max_zeros_batch(sets[:8], td)
    t0 = time.perf_counter()
    res = o.max_zeros_batch(sets, td)
    dt = time.perf_counter() - t0
    passed = sum(1 for r in res if r <= 49 - td)
    return {"workload": f"{n} seeded sets, k=15, target_distance={td}",
            "seconds": dt, "codes_per_s": n / dt, "passed": passed,
            "reference_equivalent_messages_if_exhaustive": float(n * (8 ** 15 - 1))}


def mutation_stream(n: int, seed: int, k_lo: int = 10, k_hi: int = 15):
    """n requests: single-point mutations (add / remove / move one exponent)
    of 256 seeded parents with |P| in k_lo..k_hi."""
    rng = np.random.default_rng(seed)
    parents = [sorted(rng.choice(49, int(rng.integers(k_lo, k_hi + 1)), replace=False).tolist())
               for _ in range(256)]
    out = []
    for _ in range(n):
        p = list(parents[int(rng.integers(len(parents)))])
        free = [x for x in range(49) if x not in p]
        op = int(rng.integers(3))
        if op == 0 and len(p) < k_hi:
            p.append(int(rng.choice(free)))
        elif op == 1 and len(p) > k_lo:
            p.pop(int(rng.integers(len(p))))
        else:
            p[int(rng.integers(len(p)))] = int(rng.choice(free))
        out.append(sorted(p))
    return out


def bench_served(dev: int, n: int = 3000, rate: float = 300.0, engine: str = "batch") -> dict:
    """Served search stream: Poisson arrivals at `rate` per second of mutated
    candidates, each with the running best-known d of its k as threshold.
    engine "batch": ToricBatchServer (continuous micro-batches of the batch
    path); "persistent": ToricServer (the device-resident request loop)."""
    from generalized_toric_gpu_search_b200.serve import ToricBatchServer, ToricServer

    stream = mutation_stream(n, BASE_SEED + 7)
    rng = np.random.default_rng(BASE_SEED + 11)
    gaps = rng.exponential(1.0 / rate, size=n)
    best = {k: FALLBACK_BEST_D.get(k, 1) for k in range(10, 16)}
    import threading

    lock = threading.Lock()

    def on_done(fut, k):
        a = fut.result()
        if a.passed:
            with lock:
                if a.min_distance > best[k]:
                    best[k] = a.min_distance

    make = (lambda: ToricBatchServer(dev, k_max=15)) if engine == "batch" else \
        (lambda: ToricServer(dev, k_max=15))
    with make() as srv:
        srv.evaluate([(s, best[len(s)]) for s in stream[:32]])  # warm the loop
        futs = []
        t0 = time.perf_counter()
        t_next = t0
        for s, gap in zip(stream, gaps):
            t_next += gap
            # Sleep (which releases the GIL for the server's threads) rather
            # than spin until the arrival time.
            while True:
                wait = t_next - time.perf_counter()
                if wait <= 0.0:
                    break
                time.sleep(wait)
            with lock:
                td = best[len(s)]
            f = srv.submit(s, td)
            f.add_done_callback(lambda fut, k=len(s): on_done(fut, k))
            futs.append(f)
        answers = [f.result(timeout=600) for f in futs]
        total = time.perf_counter() - t0
        st = srv.stats()
        slots = getattr(srv, "slots", None)
        # Saturation: a second stream of the same size submitted at once.
        burst = mutation_stream(n, BASE_SEED + 13)
        tb = time.perf_counter()
        srv.evaluate([(s, best[len(s)]) for s in burst], timeout=600)
        burst_s = time.perf_counter() - tb
    # The plain form on the same burst: one max_zeros call (one batch of one
    # code) per request, in arrival order, on a prefix of the stream.
    from generalized_toric_gpu_search_b200.distance import DistanceOracleCUDABP
    from generalized_toric_gpu_search_b200.tables import build_eval_matrix

    plain_o = DistanceOracleCUDABP(dev, build_eval_matrix())
    n_plain = min(n, 500)
    plain_o.max_zeros(burst[0], best[len(burst[0])])
    tp = time.perf_counter()
    for s in burst[:n_plain]:
        plain_o.max_zeros(s, best[len(s)])
    plain_s = time.perf_counter() - tp
    lat = np.array([a.latency_s for a in answers])
    dev_t = np.array([a.device_s for a in answers])
    return {"workload": (f"{n:,} Poisson arrivals at {rate:.0f}/s, single mutations of 256 seeded "
                         "parents, |P| 10..15, td = running best-known d per k"),
            "engine": engine,
            "codes_per_s": n / total, "seconds": total,
            "p50_ms": 1e3 * float(np.percentile(lat, 50)),
            "p99_ms": 1e3 * float(np.percentile(lat, 99)),
            "device_p50_ms": 1e3 * float(np.percentile(dev_t, 50)),
            "device_p99_ms": 1e3 * float(np.percentile(dev_t, 99)),
            "dedup_answers": st["dedup_answers"], "passed": int(sum(a.passed for a in answers)),
            "slots": slots, "loop_launches": st.get("loop_launches"),
            "batches": st.get("batches"),
            "burst_codes_per_s": n / burst_s,
            "plain_one_code_per_call_codes_per_s": n_plain / plain_s,
            "burst_vs_plain": (n / burst_s) / (n_plain / plain_s),
            "plain_sample": f"first {n_plain} requests of the burst, one max_zeros call each",
            "best_known_d_end": best}


# ---------------------------------------------------------------------------
# B200 arm
# ---------------------------------------------------------------------------

def measure_pipes(device: int) -> dict:
    import ctypes

    import torch

    from generalized_toric_gpu_search_b200 import _lib

    scratch = torch.empty(1 << 20, dtype=torch.uint8, device=f"cuda:{device}")
    out = (ctypes.c_double * 6)()
    _lib.check(_lib.load().tg_measure_int_pipes(device, scratch.data_ptr(), out),
               "tg_measure_int_pipes")
    return {"lop3_per_clk_sm": out[0], "popc_per_clk_sm": out[1], "iadd_per_clk_sm": out[2],
            "addmax_per_clk_sm": out[3], "lop3_popc_mix_per_clk_sm": out[4],
            "ubench_sm_mhz": out[5]}


def run_b200_arm(args, d: Dist) -> None:
    import torch

    from generalized_toric_gpu_search_b200 import _lib
    from generalized_toric_gpu_search_b200 import build as lib_build
    from generalized_toric_gpu_search_b200.distance import (
        DistanceOracleCUDABP,
        DistanceRunner,
        LaunchConfig,
        ToricContext,
        pack_sets,
    )
    from generalized_toric_gpu_search_b200.tables import build_eval_matrix

    if not torch.cuda.is_available():
        raise SystemExit("bench.py needs a CUDA device")
    lib_build.build()
    dev = d.local_rank if d.world > 1 else 0
    torch.cuda.set_device(dev)
    device = torch.device("cuda", dev)
    d.init("nccl")
    sets = make_workload(d.rank, args.n_sets, args.kmin, args.kmax)
    M = build_eval_matrix()
    ctx = ToricContext(dev, M)
    flat, offsets, kmax = pack_sets(sets)
    # Exact batches of the toric matrix (k >= 2) take the toric walk, whose shape
    # is fixed.  The walks over all messages take the shape that a table of this
    # device holds for the batch's largest k, with the command line's overrides.
    from dataclasses import asdict, replace

    from generalized_toric_gpu_search_b200 import autotune

    toric_walk = takes_toric_walk(kmax, args.enumeration)
    tuned = None
    if not toric_walk and not args.no_autotune:
        tuned = autotune.choose(autotune.load_table(_lib.device_info(dev)[3]), kmax)
    cfg = replace(tuned or LaunchConfig(), enumeration=ENUMERATIONS[args.enumeration][0])
    if args.tail_rows:
        cfg = replace(cfg, tail_rows=args.tail_rows)
    if args.blocks_per_sm:
        cfg = replace(cfg, blocks_per_sm=args.blocks_per_sm)
    runner = DistanceRunner(ctx, cfg)
    d_idx = torch.from_numpy(flat).to(device)
    d_off = torch.from_numpy(offsets).to(device)
    d_out = torch.empty(len(sets), dtype=torch.int32, device=device)
    p = runner.params(len(sets), kmax, 1)
    ws = runner.workspace(p)
    stream = torch.cuda.Stream(device=device)
    flush = torch.empty(L2_FLUSH_BYTES, dtype=torch.uint8, device=device)

    # CUDA graphs for the preparation (header resets, prep; scans of the general
    # walk), the walk over all messages (which a toric batch does not have) and
    # the information-set walk, so each is timed by its own events.
    g_prep, g_enum, g_is = (torch.cuda.CUDAGraph() for _ in range(3))
    with torch.cuda.stream(stream):
        runner.run(p, d_idx, d_off, d_out, stream=stream, workspace=ws)  # warm the module
    stream.synchronize()
    with torch.cuda.graph(g_prep, stream=stream, capture_error_mode="thread_local"):
        runner.prepare(p, d_idx, d_off, d_out, stream=stream, workspace=ws)
    def walk_graph(graph, parts):
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            runner.walk(p, d_out, stream=stream, workspace=ws, parts=parts)
        return graph.replay

    def no_walk():
        pass

    if toric_walk:
        enum_replay, is_replay = no_walk, walk_graph(g_is, _lib.TG_WALK_INFOSET)
    else:  # no set of such a batch is left to information sets
        enum_replay, is_replay = walk_graph(g_enum, _lib.TG_WALK_ENUMERATION), no_walk

    def step():
        g_prep.replay()
        enum_replay()
        is_replay()

    with torch.cuda.stream(stream):
        for _ in range(args.warmup):
            step()
    stream.synchronize()
    check = d_out.cpu().tolist()
    tasks, codewords, ref_msgs = runner.counters(stream)
    paths = runner.path_counters(stream)
    stages = runner.stage_counters(stream)
    with torch.cuda.stream(stream):
        g_prep.replay()  # what the preparation evaluates by itself
    prep_codewords = runner.path_counters(stream)["infoset_codewords"]

    ev = [[torch.cuda.Event(enable_timing=True) for _ in range(4)] for _ in range(args.steps)]
    clocks = clock_sampler(dev)
    d.barrier()
    torch.cuda.synchronize()
    clocks.start()
    with torch.cuda.stream(stream):
        for i in range(args.steps):
            flush.zero_()  # L2 flush between steps, outside the events
            ev[i][0].record(stream)
            g_prep.replay()
            ev[i][1].record(stream)
            enum_replay()
            ev[i][2].record(stream)
            is_replay()
            ev[i][3].record(stream)
    # Wait with the GIL released, so the clock sampler's thread keeps sampling
    # through the timed region (the step times come from the CUDA events).
    while not ev[-1][3].query():
        time.sleep(0.0005)
    stream.synchronize()
    torch.cuda.synchronize()
    clk = clocks.stop()
    d.barrier()
    step_ms = [e[0].elapsed_time(e[3]) for e in ev]
    prep_ms = [e[0].elapsed_time(e[1]) for e in ev]
    enum_ms = [e[1].elapsed_time(e[2]) for e in ev]
    is_ms = [e[2].elapsed_time(e[3]) for e in ev]
    if d_out.cpu().tolist() != check:
        raise SystemExit("results changed between steps")
    total_ms = d.max(sum(step_ms), device)
    all_ref = d.sum(ref_msgs, device)
    value = all_ref / (total_ms / 1e3 / args.steps)

    # End to end through the public API: host lists in, host list out.
    oracle = DistanceOracleCUDABP(dev, M, cfg)
    for _ in range(args.warmup):  # full-size calls: workspace and pinned buffers at size
        oracle.max_zeros_batch(sets, 1)
    h2d = flat.nbytes + offsets.nbytes
    d2h = 4 * len(sets)
    e2e_s = []
    d.barrier()
    for _ in range(args.steps):
        t0 = time.perf_counter()
        res = oracle.max_zeros_batch(sets, 1)
        e2e_s.append(time.perf_counter() - t0)
    if res != check:
        raise SystemExit("public API result differs from the device-resident run")
    e2e_max = d.max(sum(e2e_s), device)
    e2e_value = all_ref / (e2e_max / args.steps)

    # Plain one-code-per-launch form on a stratified sample (same kernels).
    plain = None
    if d.rank == 0 and not args.skip_plain:
        sample = stratified_sample(sets, 4)
        hist = k_histogram(sets)
        t_k = {}
        for k, group in sample.items():
            times = []
            for s in group:
                fl, of, km = pack_sets([s])
                di, do = torch.from_numpy(fl).to(device), torch.from_numpy(of).to(device)
                dd = torch.empty(1, dtype=torch.int32, device=device)
                pp = runner.params(1, km, 1)
                wws = torch.empty(max(int(1 << 20), 256), dtype=torch.uint8, device=device)
                e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                with torch.cuda.stream(stream):
                    e0.record(stream)
                    runner.run(pp, di, do, dd, stream=stream, workspace=wws)
                    e1.record(stream)
                stream.synchronize()
                times.append(e0.elapsed_time(e1) / 1e3)
            t_k[k] = statistics.mean(times)
        plain_s = sum(hist[k] * t_k[k] for k in hist)
        plain = {"value": ref_msgs / plain_s, "unit": UNIT, "codes_per_s": len(sets) / plain_s,
                 "sample": "4 sets per k, one launch per set, per-k mean time x k histogram"}

    pipes = measure_pipes(dev) if d.rank == 0 else {}
    mhz = clk.get("sm_mhz") or pipes.get("ubench_sm_mhz") or 1965.0
    roof = roofline(toric_walk, statistics.mean(prep_ms) / 1e3, statistics.mean(enum_ms) / 1e3,
                    statistics.mean(is_ms) / 1e3, prep_codewords, paths, pipes, ctx.sm_count, mhz)

    extra = {}
    ref_gpu = None
    if d.rank == 0 and not args.skip_plain:
        ref_gpu = bench_reference_gpu(dev, sets)
    if d.rank == 0 and not args.skip_extra:
        extra["canonical_forms"] = bench_canonical(dev)
        extra["early_exit_k15"] = bench_early_exit(dev)
        extra["served_stream"] = bench_served(dev, engine="persistent")
        extra["served_stream_batch"] = bench_served(dev, engine="batch")

    cpu = None
    if d.rank == 0 and d.world == 1 and not args.skip_cpu:
        cpu = cpu_reference_rate(sets, 1 << 26, per_k=4)

    if d.rank == 0:
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": d.world,
            "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": total_ms / args.steps, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "u32 bit-sliced GF(8) (integer LOP3/POPC)",
            "data": "synthetic (seeded random exponent sets)",
            "config": {"workload": WORKLOAD, "n_sets_per_gpu": len(sets),
                       "k_range": [K_LO, K_HI], "target_distance": 1,
                       "enumeration": ENUMERATIONS[args.enumeration][1],
                       "variant": "toric walk" if toric_walk else "histogram",
                       "tail_rows": None if toric_walk else args.tail_rows or 4,
                       "launch": "CUDA graphs: preparation, toric walk" if toric_walk else
                                 "CUDA graphs: preparation, walk over all messages",
                       "launch_shape": {k_: v for k_, v in asdict(cfg).items()
                                        if k_ not in ("enumeration", "variant")},
                       "launch_shape_source":
                           "fixed: toric walk, two CTAs per SM" if toric_walk else
                           "table of this device for k = %d (0 = library default)" % kmax
                           if tuned else "library defaults",
                       "l2": "256 MiB write between timed steps",
                       "parallelism": f"weak, {d.world} rank(s), no data-path collective"},
            "codes_per_s": d.world * len(sets) / (total_ms / 1e3 / args.steps),
            "evaluated_codewords_per_s": d.world * codewords / (total_ms / 1e3 / args.steps),
            "evaluated_codewords_per_step": codewords, "path_counters": paths,
            "infoset_codewords_by_stage": stages,
            "prep_ms": statistics.mean(prep_ms), "enumeration_walk_ms": statistics.mean(enum_ms),
            "infoset_walk_ms": statistics.mean(is_ms),
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": int(h2d),
                    "d2h_bytes_per_step": int(d2h), "ms_per_step": 1e3 * e2e_max / args.steps,
                    "api": "DistanceOracleCUDABP.max_zeros_batch(list of lists, 1)"},
            "gpu_launches": step_launches(kmax, args.enumeration) * args.steps,
            "roofline": roof,
            "int_pipes": pipes,
            "clocks": clk,
            "plain_form": plain,
            "batched_vs_plain": (value / plain["value"]) if plain else None,
            "reference_gpu": ref_gpu,
            "batched_vs_reference_gpu": (value / ref_gpu["batched_per_k_launch"]["value"])
            if ref_gpu and "batched_per_k_launch" in ref_gpu else None,
            "batched_vs_reference_gpu_one_per_launch":
                (value / ref_gpu["one_code_per_launch"]["value"])
                if ref_gpu and "one_code_per_launch" in ref_gpu else None,
            # the reference's enumeration (all 8^k - 1 messages) on the B200 and on
            # the host cores: a hardware-only ratio of the same algorithm
            "same_algorithm_gpu_vs_cpu": (ref_gpu["batched_per_k_launch"]["value"] / cpu["value"])
            if ref_gpu and "batched_per_k_launch" in ref_gpu and cpu else None,
            "cpu_baseline": cpu,
            **extra,
        }
        print(json.dumps(line), flush=True)
    del g_prep, g_enum, g_is
    d.close()


def main(argv=None) -> None:
    ap = argparse.ArgumentParser(description=__doc__.splitlines()[0])
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["b200", "reference"], default="b200")
    ap.add_argument("--tail-rows", type=int, default=0)
    ap.add_argument("--blocks-per-sm", type=int, default=0)
    ap.add_argument("--enumeration", choices=sorted(ENUMERATIONS), default="auto",
                    help="exact enumeration of the headline workload")
    ap.add_argument("--skip-plain", action="store_true")
    ap.add_argument("--no-autotune", action="store_true",
                    help="library default launch shapes instead of the tuned ones")
    ap.add_argument("--skip-cpu", action="store_true")
    ap.add_argument("--skip-extra", action="store_true",
                    help="skip the canonical, early-exit and served-stream sections")
    ap.add_argument("--n-sets", type=int, default=N_SETS, help="sets per GPU (small cases)")
    ap.add_argument("--kmin", type=int, default=K_LO)
    ap.add_argument("--kmax", type=int, default=K_HI)
    ap.add_argument("--section", choices=["canonical", "early-exit", "served", "served-persistent",
                                          "reference-gpu"],
                    help="run one secondary configuration alone and print its JSON")
    ap.add_argument("--canon-n", type=int, default=1_000_000)
    args = ap.parse_args(argv)
    d = Dist()
    if args.section:
        from generalized_toric_gpu_search_b200 import build as lib_build

        lib_build.build()
        fn = {"canonical": lambda: bench_canonical(0, args.canon_n),
              "early-exit": lambda: bench_early_exit(0),
              "served": lambda: bench_served(0, engine="batch"),
              "served-persistent": lambda: bench_served(0, engine="persistent"),
              "reference-gpu": lambda: bench_reference_gpu(0, make_workload(0))}[args.section]
        print(json.dumps({"section": args.section, **fn()}), flush=True)
        return
    if args.impl == "reference":
        run_reference_arm(args, d)
        return
    run_b200_arm(args, d)


if __name__ == "__main__":
    main()
