#!/usr/bin/env python
"""Benchmark: Poseidon2 permutations proven per second with the B200 Whirlaway prover.

A step is one plain proof of the Poseidon2-KoalaBear width-16 AIR over 2^log_n
permutations (one per trace row; default 2^20, the plain-at-scale configuration) with the
reference's default parameters (rate 1/2, folding 7 then 4, univariate skip 4, 128-bit
security, 16 PoW bits). Inputs are uniform KoalaBear elements from StdRng in the
reference's draw order (synthetic, as in the reference example).

  value  throughput with the witness resident in HBM (AirTable::prove on a device witness)
  e2e    the same through the C ABI from the permutation inputs in pinned host memory: every step
         copies the 16 inputs per row to the device, generates the trace there
         (wl_witness_generate) and proves it, and the proof comes back to the host; the copies
         and the trace generation are inside the timed region
  e2e_host_witness  the same with the whole witness (165 columns) in pinned host memory
         instead (wl_prove: its host-to-device copy overlaps the first commitment)

N > 1 GPUs: one process per GPU (torchrun), each proving its own independent instances
(replicas: proofs share nothing, so there is no collective on the data path); the timed
region is bracketed by a barrier and the maximum over ranks is reported.

--impl reference runs the CPU restatement of the reference prover (the oracle; the Rust
reference cannot be built here) with all host threads on a bounded sample of the workload.
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "Poseidon2 perms proven/sec on 1 B200 (batched vs plain); p50/p99 proof latency"
# field products on the CUDA cores: the S-boxes (the partial rounds' linear layers and, in the
# zerocheck's round 0, the extension and the weights run on the tensor cores)
P24_MODMUL = 8 * 24 * 2 + 23 * 2
P16_MODMUL = 8 * 16 * 2 + 20 * 2
ZC0_MODMUL_PER_POINT = 148 * 2


def parse_args():
    ap = argparse.ArgumentParser(description=__doc__, formatter_class=argparse.RawDescriptionHelpFormatter)
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--log-n", type=int, default=20)
    ap.add_argument("--cpu-sample-log-n", type=int, default=15,
                    help="trace height of the bounded CPU-baseline sample")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-e2e", action="store_true")
    ap.add_argument("--no-batched", action="store_true")
    ap.add_argument("--no-serving", action="store_true")
    ap.add_argument("--batch-size", type=int, default=64)
    ap.add_argument("--workers", type=int, default=16)
    ap.add_argument("--no-sumcheck", action="store_true")
    ap.add_argument("--sumcheck-log-n", type=int, default=24)
    ap.add_argument("--sumcheck-reps", type=int, default=3)
    ap.add_argument("--serving-requests", type=int, default=2000, help="requests per arrival rate")
    ap.add_argument("--serving-rates", type=str, default="1,4",
                    help="offered load as multiples of the plain path's capacity on the mix")
    return ap.parse_args()


def workload_config(log_n):
    return {
        "workload": f"plain single proof, Poseidon2-KoalaBear width-16 AIR, 2^{log_n} permutations (one per row)",
        "log_n_rows": log_n,
        "air_columns": 165,
        "whir": "rate 1/2, folding 7 then 4, RS domain reduction 2^5, 16 PoW bits, 128-bit CapacityBound",
        "univariate_skips": 4,
        "extension": "KoalaBear^8 (X^8 - 3)",
        "inputs": "uniform KoalaBear from StdRng, reference draw order",
        "l2": "inputs larger than L2 (witness 165 x 2^log_n x 4 B, LDE 88 x 2^(log_n+2) x 4 B)",
        "parallelism": "replicas",
    }


# ----------------------------------------------------------------------------- clocks
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    INTERVAL_MS = 20  # several samples inside a timed region of a few proofs

    def __init__(self, device):
        self.device = device
        self.proc = None
        self.path = None
        self.skip = 0
        self.interval_ms = self.INTERVAL_MS

    def _lines(self):
        with open(self.path) as f:
            return f.read().split("\n")[:-1]  # complete lines only

    def start(self):
        fd, self.path = tempfile.mkstemp(suffix=".csv")
        os.close(fd)
        # the short interval first; should nvidia-smi refuse it, the next one
        for interval in (self.INTERVAL_MS, 100):
            try:
                self.proc = subprocess.Popen(
                    ["nvidia-smi", "-i", str(self.device), f"--query-gpu={self.FIELDS}", "--format=csv,noheader",
                     "-lms", str(interval)], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
            except OSError:
                self.proc = None
                return
            self.interval_ms = interval
            # nvidia-smi's start-up (driver and NVML initialisation) must not overlap the timed
            # region: wait for its first sample line before returning; the lines written so far
            # precede the region and are left out
            t0 = time.time()
            while time.time() - t0 < 5.0 and self.proc.poll() is None:
                if os.path.getsize(self.path) > 0 and self._lines():
                    break
                time.sleep(0.005)
            if self._lines() or self.proc.poll() is None:
                break
        self.skip = len(self._lines())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        lines = self._lines()
        os.unlink(self.path)
        in_region = lines[self.skip:]
        # a region shorter than the interval has no sample of its own: the one just before it
        use = in_region if in_region else lines[-1:]
        sm, smax, reasons, power = [], [], set(), []
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in use:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1].split()[0]))
                smax.append(float(parts[2].split()[0]))
                power.append(float(parts[3].split()[0]))
            except ValueError:
                continue
            for n, v in zip(names, parts[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        return {"sm_mhz": statistics.median(sm) if sm else None, "sm_max_mhz": max(smax) if smax else None,
                "reasons": sorted(reasons), "samples": len(sm), "samples_in_region": bool(in_region),
                "interval_ms": self.interval_ms, "power_w_max": max(power) if power else None}


# ----------------------------------------------------------------------------- distributed
def dist_setup(args):
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if world > 1:
        import datetime
        import torch
        import torch.distributed as dist
        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=600),
                                device_id=torch.device("cuda", local))
    return world, rank, local


def dist_max(value, world):
    """Maximum of a per-rank value over all ranks (the job time of a replica run)."""
    if world == 1:
        return value
    import torch
    import torch.distributed as dist
    device = "cuda" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([value], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def replica_input_seed(world, rank):
    """Input stream of a replica: the reference's single stream alone, one seed per rank otherwise."""
    return -1 if world == 1 else rank


def barrier(world):
    if world > 1:
        import torch.distributed as dist
        dist.barrier()


# ----------------------------------------------------------------------------- CPU arm
def cpu_prove_rate(log_n, steps, warmup, threads=None):
    """The oracle (CPU restatement of the reference prover) on 2^log_n rows: perms/s."""
    from tests import oracle_lib
    oracle = oracle_lib.load()
    if threads:
        oracle.lib.wlo_set_threads(threads)
    cores = oracle.lib.wlo_max_threads()
    consts, inputs = oracle.workload(log_n)
    wit = oracle.trace(log_n, consts, inputs)
    for _ in range(warmup):
        oracle.prove(log_n, consts, wit)
    t0 = time.perf_counter()
    for _ in range(steps):
        proof, _ = oracle.prove(log_n, consts, wit)
    dt = time.perf_counter() - t0
    assert oracle.verify(log_n, consts, proof) == 0
    return steps * (1 << log_n) / dt, cores, dt / steps


def cpu_model():
    """The host CPU's model name (from /proc/cpuinfo), for the baseline record."""
    try:
        with open("/proc/cpuinfo") as f:
            for line in f:
                if line.startswith("model name"):
                    return line.split(":", 1)[1].strip()
    except OSError:
        pass
    return "unknown"


def run_reference(args, world, rank):
    if rank != 0:
        return
    log_n = min(args.cpu_sample_log_n, args.log_n)
    rate, cores, sec = cpu_prove_rate(log_n, args.steps, args.warmup)
    sample = (f"CPU oracle (restatement of the reference prover, {cores} threads) proving 2^{log_n} rows per step; "
              f"{sec:.2f} s per step")
    print(json.dumps({
        "impl": "reference", "metric": METRIC, "value": rate, "unit": "perms/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u32 (KoalaBear Montgomery)", "data": "synthetic",
        "config": workload_config(args.log_n),
        "cpu_baseline": {"value": rate, "unit": "perms/s", "cores": cores, "kind": "port", "sample": sample,
                         "cpu_model": cpu_model(), "nproc": os.cpu_count()},
        "e2e": {"value": rate, "unit": "perms/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }), flush=True)


# ----------------------------------------------------------------------------- GPU arm
def int_peaks(device, consts):
    """Integer-pipe throughput of the device from the benchmark's probe library, all from
    registers: raw 32-bit multiplies (mul.lo/s, mul.hi/s), Montgomery products/s and
    Poseidon2-24 permutations/s."""
    import ctypes
    import numpy as np
    lib = ctypes.CDLL(os.path.join(ROOT, "whirlaway_b200", "_build", "libwl_probe.so"))
    a, b, lo, hi = ctypes.c_double(), ctypes.c_double(), ctypes.c_double(), ctypes.c_double()
    c = np.ascontiguousarray(consts, dtype=np.uint32)
    rc = lib.wlp_int_peaks(device, c.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), ctypes.byref(a), ctypes.byref(b))
    rc = rc or lib.wlp_mul_peaks(device, ctypes.byref(lo), ctypes.byref(hi))
    if rc:
        raise RuntimeError(f"integer-peak probe failed with CUDA error {rc}")
    return {"mul_lo_per_s": lo.value, "mul_hi_per_s": hi.value, "modmul_per_s": a.value, "p24_perms_per_s": b.value}


LEAF_EXTRA_DRAM_BYTES = 26.1  # measured DRAM bytes per leaf row beyond the row itself (k_leaf_hash)


def whir_rows_hashed(log_n):
    """Leaf rows hashed per proof (all WHIR commitments) under the default parameters."""
    m = log_n + 8
    ld = m + 1
    rows = [1 << (ld - 7)]
    rest = m - 7
    rounds = 0 if rest < 6 else (rest - 6 + 3) // 4
    ld -= 5
    m -= 7
    for _ in range(rounds):
        rows.append(1 << (ld - 4))
        ld -= 1
        m -= 4
    return rows


def read_hbm_peak():
    """The HBM copy peak (GB/s) the roofline is measured against, and where it comes from: the
    measured figure in MEASURED_PEAKS.json when the file is there, else a fallback of 6.65 TB/s
    (a STREAM-style copy measured earlier on a B200)."""
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            return float(json.load(f)["hbm_gbs"]), "MEASURED_PEAKS.json hbm_gbs (measured)"
    except (OSError, KeyError, ValueError, TypeError):
        return 6650.0, "fallback: 6.65 TB/s, a copy measured earlier on a B200 (MEASURED_PEAKS.json absent)"


def roofline(profile, breakdown, log_n, peaks, hbm_peak_gbs, steps, hbm_source):
    """Roofline of the dominant kernel class: its CUDA-event time over the timed region
    (`profile`), its share of all kernel time from a fully profiled proof (`breakdown`)."""
    name, (ms, launches) = max(profile.items(), key=lambda kv: kv[1][0])
    N = 1 << log_n
    rows = whir_rows_hashed(log_n)
    per_launch_ms = ms / max(launches, 1)
    out = {"kernel": name, "launches": launches, "avg_launch_ms": per_launch_ms,
           "share_of_kernel_time": breakdown[name][0] / sum(v[0] for v in breakdown.values())}
    # hardware ceiling of field multiplication: a Montgomery product needs two low-word and two
    # high-word 32-bit multiplies; the raw multiply rates come from dependency-free probes
    modmul_peak = 1.0 / (2.0 / peaks["mul_lo_per_s"] + 2.0 / peaks["mul_hi_per_s"])
    if name == "merkle_tree":
        # leaf sponges (8 Poseidon2-24 per row) and 2-to-1 compressions (Poseidon2-16, counted
        # as Poseidon2-24 equivalents by their share of field multiplications)
        perms = (sum(rows) * 8 + sum(rows) * P16_MODMUL / P24_MODMUL) * steps
        byts = (rows[0] * (88 * 4 + 64) + sum(r * (128 * 4 + 64) for r in rows[1:])) * steps
        achieved = perms * P24_MODMUL / (ms * 1e-3)
        # DRAM traffic per Merkle build: ncu's dram__bytes_read.sum + dram__bytes_write.sum of the
        # leaf kernel is 378.1 B per row on 2^19 leaf rows of 88 columns, 184 MB (the row once plus
        # 26.1 B, most of them the digest); scaled by rows, with 128-column rows for the later
        # commitments. The compressions' own traffic is not in it.
        traffic = (rows[0] * (88 * 4 + LEAF_EXTRA_DRAM_BYTES)
                   + sum(r * (128 * 4 + LEAF_EXTRA_DRAM_BYTES) for r in rows[1:])) * steps / max(launches, 1)
        out.update({"bound": "int", "achieved": achieved / 1e12, "peak": modmul_peak / 1e12,
                    "unit": "T S-box products/s (430 per Poseidon2-24; the partial rounds' linear layers run on the tensor cores)",
                    "frac": achieved / modmul_peak, "traffic": traffic,
                    "traffic_source": "ncu counters of k_leaf_hash on 2^19 leaf rows of 88 columns (378.1 B a row), "
                                      "scaled by rows",
                    "frac_note": "the S-boxes are four low-word multiplies and four fp64 operations each, so this is "
                                 "work done against the integer pipe's rate, not the distance from what binds the "
                                 "kernel: its S-boxes' register reads, 14 to 15 clocks a warp and scheduler",
                    "peak_source": ("hardware: 32-bit multiplies measured in this run by dependency-free mul.lo / "
                                    "mul.hi probes, two of each per Montgomery product"),
                    "p24_per_s": perms / (ms * 1e-3),
                    "same_code_probe_view": {"achieved": perms / (ms * 1e-3) / 1e9,
                                             "peak": peaks["p24_perms_per_s"] / 1e9, "unit": "G Poseidon2-24 perms/s",
                                             "frac": perms / (ms * 1e-3) / peaks["p24_perms_per_s"],
                                             "note": "against back-to-back permutations of the one-thread form "
                                                     "from registers (no tensor cores)"},
                    "hbm": {"achieved": byts / (ms * 1e-3) / 1e9, "peak": hbm_peak_gbs, "unit": "GB/s",
                            "frac": byts / (ms * 1e-3) / 1e9 / hbm_peak_gbs,
                            "peak_source": hbm_source}})
        return out
    if name == "leaf_hash":
        work = sum(rows) * 8 * P24_MODMUL * steps
        byts = (rows[0] * (88 * 4 + 32) + sum(r * (128 * 4 + 32) for r in rows[1:])) * steps
    elif name == "zc0_eval":
        work = (N >> 4) * 30 * ZC0_MODMUL_PER_POINT * steps
        byts = 165 * N * 4 * steps
    elif name == "merkle":
        work = sum(rows) * P16_MODMUL * steps
        byts = sum(rows) * 2 * 32 * steps
    else:
        work, byts = None, None
    if work is not None:
        achieved = work / (ms * 1e-3) / 1e9
        peak = modmul_peak / 1e9
        out.update({"bound": "int", "achieved": achieved, "peak": peak, "unit": "Gmodmul/s",
                    "frac": achieved / peak, "traffic": None,
                    "peak_source": "hardware: 32-bit multiplies (mul.lo / mul.hi probes), two of each per Montgomery product",
                    "hbm": {"achieved": byts / (ms * 1e-3) / 1e9, "peak": hbm_peak_gbs, "unit": "GB/s",
                            "frac": byts / (ms * 1e-3) / 1e9 / hbm_peak_gbs,
                            "peak_source": hbm_source}})
    return out


def batched_run(wl, args):
    """Batched configuration: independent proofs with log2 rows ~ U{12..18} (seed 0), each with
    its own input stream and transcript, concurrently on one device, against the same mix
    proved one at a time on one stream."""
    import numpy as np
    rng = np.random.default_rng(0)
    sizes = [int(x) for x in rng.integers(12, 19, args.batch_size)]
    jobs = [(*wl.generate_workload(n, 1000 + k), n) for k, n in enumerate(sizes)]
    rows = sum(1 << n for n in sizes)
    with wl.Server(0, workers=args.workers, hbm_budget_bytes=160 << 30) as srv:
        # one untimed pass of the whole mix: the stream-ordered pool grows to the mix's peak
        # footprint (16 streams' worth of buffers) before the timed pass
        wl.batch_prove(srv, jobs)
        t0 = time.perf_counter()
        proofs = wl.batch_prove(srv, jobs)
        batched_s = time.perf_counter() - t0
    with wl.Context(0) as ctx:
        tables = []
        for c, i, n in jobs[:2]:
            w = wl.Witness.generate(ctx, c, i, n)
            wl.AirTable(ctx, c, n).prove_witness(w)
            w.free()
        t0 = time.perf_counter()
        plain = []
        for c, i, n in jobs:
            w = wl.Witness.generate(ctx, c, i, n)
            plain.append(wl.AirTable(ctx, c, n).prove_witness(w))
            w.free()
        plain_s = time.perf_counter() - t0
    same = all(np.array_equal(a, b) for a, b in zip(proofs, plain))
    # the batch's proofs verified by the library: host threads only, and with the Merkle paths
    # of all proofs checked in one GPU kernel (the transcripts replay on host threads)
    consts = jobs[0][0]
    assert all(np.array_equal(c, consts) for c, _, _ in jobs)
    vjobs = [(n, p) for (_, _, n), p in zip(jobs, proofs)]
    t0 = time.perf_counter()
    st_host = wl.verify_batch(consts, vjobs)
    verify_host_s = time.perf_counter() - t0
    with wl.Context(0) as vctx:
        wl.verify_batch_device(vctx, consts, vjobs[:4])  # warm-up
        t0 = time.perf_counter()
        st_dev = wl.verify_batch_device(vctx, consts, vjobs)
        verify_dev_s = time.perf_counter() - t0
    verify = {"proofs": len(vjobs), "all_accepted": bool(all(x == 0 for x in st_host) and st_dev == st_host),
              "host_threads_ms": verify_host_s * 1e3, "gpu_merkle_ms": verify_dev_s * 1e3,
              "timing": "host wall clock over the batch"}
    return {"proofs": len(jobs), "verify": verify, "log_n_rows": "U{12..18}, seed 0", "workers": args.workers,
            "value": rows / batched_s, "unit": "perms/s", "wall_s": batched_s,
            "plain_one_at_a_time_perms_per_s": rows / plain_s, "speedup_vs_plain": plain_s / batched_s,
            "byte_identical_to_plain": bool(same),
            "timing": "host wall clock around submit-all/wait-all, inputs on the host (trace generated on the GPU)"}


def sumcheck_run(wl, ctx, args):
    """Sumcheck + folding microbench: the zerocheck of eq(r, x) * (a(x) b(x) - c(x)) over three
    columns of 2^24 base-field values (a, b uniform from a seed, c = a * b so that the
    constraint vanishes), with the first round univariate-skipping 3 variables; per-round times
    (CUDA events on the library's stream, from the round's first launch to its fold, host
    transcript work between them included) and each round's algorithmic HBM bytes."""
    import numpy as np
    import torch
    log_n, k = args.sumcheck_log_n, 3
    gen = torch.Generator(device="cuda").manual_seed(7)
    p = 0x7F000001
    a = torch.randint(0, p, (1 << log_n,), generator=gen, device="cuda", dtype=torch.int64)
    b = torch.randint(0, p, (1 << log_n,), generator=gen, device="cuda", dtype=torch.int64)
    c = (a * b) % p
    a, b, c = (x.to(torch.int32) for x in (a, b, c))
    consts, _ = wl.generate_workload(2)
    p16 = consts[148:296]
    for _ in range(2):
        proof, _ = wl.sumcheck_abc_prove(ctx, p16, log_n, k, a, b, c, device=True)
    runs = [wl.sumcheck_abc_prove(ctx, p16, log_n, k, a, b, c, device=True)[1] for _ in range(args.sumcheck_reps)]
    ctx.profile(True)  # one more run with every kernel class timed (not part of round_ms)
    wl.sumcheck_abc_prove(ctx, p16, log_n, k, a, b, c, device=True)
    prof = {n: round(v[0], 4) for n, v in ctx.profile_report().items() if not n.startswith("host:")}
    ctx.profile(False)
    rounds = [float(np.median([r[i] for r in runs])) for i in range(len(runs[0]))]
    assert wl.sumcheck_abc_verify(p16, log_n, k, proof) == 0
    S = 1 << (log_n - k)
    # round 0 writes and reads the eq table (32 B extension values) and reads a, b, c (4 B each);
    # round 1 reads them again and writes the three folded columns and the halved eq table;
    # round i >= 2 reads 3 columns of 2^(n-k-i+2) values and the eq table, and writes the halves
    byts = [3 * (1 << log_n) * 4 + 2 * S * 32, 3 * (1 << log_n) * 4 + S * 32 + 3 * S * 32 + (S // 2) * 32]
    m = log_n - k
    for i in range(1, m):
        ln = 1 << (m - i + 1)
        byts.append(3 * ln * 32 + (ln // 2) * 32 + 3 * (ln // 2) * 32 + (ln // 4) * 32)
    total = sum(rounds)
    return {"workload": f"zerocheck of eq * (a*b - c), three columns of 2^{log_n} base-field values, "
                        f"univariate skip {k}, {len(rounds)} rounds",
            "round_ms": [round(x, 4) for x in rounds], "total_ms": total,
            "round_hbm_gbs": [round(b / (t * 1e-3) / 1e9, 1) for b, t in zip(byts, rounds)],
            "round0_hbm_frac": byts[0] / (rounds[0] * 1e-3) / 1e9 / args.hbm_peak,
            "algorithmic_bytes": sum(byts), "reps": args.sumcheck_reps, "verified": True,
            "kernel_profile_ms": prof,
            "timing": "median over reps of CUDA-event time per round on the prover's stream"}


def sumcheck_cpu_baseline(args):
    """The oracle's a*b - c zerocheck on the same microbench size, all host threads."""
    import numpy as np
    from tests import oracle_lib
    oracle = oracle_lib.load()
    log_n, k = args.sumcheck_log_n, 3
    rng = np.random.default_rng(7)
    p = 0x7F000001
    a = rng.integers(0, p, 1 << log_n, dtype=np.uint64)
    b = rng.integers(0, p, 1 << log_n, dtype=np.uint64)
    c = (a * b) % p
    a, b, c = (x.astype(np.uint32) for x in (a, b, c))
    consts, _ = oracle.workload(2)
    t0 = time.perf_counter()
    oracle.prove_abc(consts[148:296], log_n, k, a, b, c)
    dt = time.perf_counter() - t0
    return {"total_ms": dt * 1e3, "cores": oracle.lib.wlo_max_threads(), "kind": "port",
            "sample": f"one oracle proof of the full microbench (2^{log_n} rows, skip {k})"}


def serving_run(wl, args):
    """Serving configuration: Poisson arrivals of requests with log2 rows log-uniform on
    [12, 20] (rounded), admitted by HBM footprint against a 160 GB budget. Offered loads are
    multiples of the plain path's capacity on this mix (proofs one at a time on one stream,
    measured on the first requests). Inputs come from a pool of four seeded instances per
    size (each request still has its own transcript and proof)."""
    import threading
    import numpy as np
    rng = np.random.default_rng(1)
    R = args.serving_requests
    sizes = [int(round(x)) for x in rng.uniform(12, 20, R)]
    pool = {n: [wl.generate_workload(n, 5000 + 16 * n + j) for j in range(4)] for n in sorted(set(sizes))}
    inputs = [pool[n][k % 4] for k, n in enumerate(sizes)]
    mean_rows = float(np.mean([1 << n for n in sizes]))
    # the plain path's rate on this mix, from its first requests proved one at a time
    sample = list(zip(inputs, sizes))[:48]
    with wl.Context(0) as ctx:
        for (c, i), n in sample[:2]:
            w = wl.Witness.generate(ctx, c, i, n)
            wl.AirTable(ctx, c, n).prove_witness(w)
            w.free()
        t0 = time.perf_counter()
        for (c, i), n in sample:
            w = wl.Witness.generate(ctx, c, i, n)
            wl.AirTable(ctx, c, n).prove_witness(w)
            w.free()
        plain_rate = sum(1 << n for _, n in sample) / (time.perf_counter() - t0)
    base = plain_rate / mean_rows  # requests/s the plain path sustains on this mix
    out = []
    with wl.Server(0, workers=args.workers, hbm_budget_bytes=160 << 30) as srv:
        wl.batch_prove(srv, [(c, i, n) for (c, i), n in list(zip(inputs, sizes))[:args.workers]])
        for mult in [float(x) for x in args.serving_rates.split(",")]:
            lam = base * mult
            gaps = rng.exponential(1.0 / lam, R)
            tickets = [None] * R
            lat = [None] * R

            def submitter():
                t_next = time.perf_counter()
                for k in range(R):
                    t_next += gaps[k]
                    d = t_next - time.perf_counter()
                    if d > 0:
                        time.sleep(d)
                    c, i = inputs[k]
                    tickets[k] = srv.submit(c, i, sizes[k])

            t0 = time.perf_counter()
            th = threading.Thread(target=submitter)
            th.start()
            done_t = 0.0
            for k in range(R):
                while tickets[k] is None:
                    time.sleep(0.0005)
                _, tm = srv.wait(tickets[k], sizes[k])
                lat[k] = tm["latency_ms"]
                done_t = time.perf_counter()
            th.join()
            wall = done_t - t0
            lat = np.array(lat)
            sustained = sum(1 << n for n in sizes) / wall
            out.append({"offered_requests_per_s": lam, "offered_x_plain_capacity": mult,
                        "sustained_perms_per_s": sustained, "sustained_x_plain": sustained / plain_rate,
                        "p50_latency_ms": float(np.percentile(lat, 50)), "p99_latency_ms": float(np.percentile(lat, 99))})
        stats = srv.stats()
    return {"requests_per_rate": R, "log_n_rows": "log-uniform on [12, 20], rounded, seed 1",
            "hbm_budget_bytes": 160 << 30, "workers": args.workers, "peak_running": stats["peak_running"],
            "peak_bytes_admitted": stats["peak_bytes_admitted"], "plain_one_at_a_time_perms_per_s": plain_rate,
            "rates": out, "timing": "host wall clock; latency = submission to proof ready"}


def run_ours(args, world, rank, local):
    import numpy as np
    import torch
    import whirlaway_b200 as wl

    torch.cuda.set_device(local)
    log_n = args.log_n
    ctx = wl.Context(local)
    consts, inputs = wl.generate_workload(log_n, replica_input_seed(world, rank))
    table = wl.AirTable(ctx, consts, log_n)
    wit = wl.Witness.generate(ctx, consts, inputs, log_n)
    peaks = int_peaks(local, consts)
    stream = torch.cuda.ExternalStream(ctx.stream_ptr)

    for _ in range(args.warmup - 1):
        table.prove_witness(wit)
    # the last warm-up proof carries the per-kernel-class breakdown; the timed region carries
    # CUDA events around the dominant class only (its launches are what the roofline divides)
    ctx.profile(True)
    table.prove_witness(wit)
    breakdown = ctx.profile_report()
    host_profile = {k[5:]: round(v[0], 4) for k, v in breakdown.items() if k.startswith("host:")}
    breakdown = {k: v for k, v in breakdown.items() if not k.startswith("host:")}
    dominant = max(breakdown.items(), key=lambda kv: kv[1][0])[0]
    sampler = ClockSampler(local)
    ctx.profile(True, only=dominant)
    syncs0, wait0 = ctx.host_syncs, ctx.host_wait_ms
    barrier(world)
    torch.cuda.synchronize()
    launches0 = wl.kernel_launch_count()
    sampler.start()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        proof = table.prove_witness(wit)
    e1.record(stream)
    e1.synchronize()
    torch.cuda.synchronize()
    clocks = sampler.stop()
    barrier(world)
    launches = wl.kernel_launch_count() - launches0
    elapsed_ms = dist_max(e0.elapsed_time(e1), world)
    profile = {k: v for k, v in ctx.profile_report().items() if not k.startswith("host:")}
    ctx.profile(False)
    host_syncs = (ctx.host_syncs - syncs0) / args.steps
    host_wait = (ctx.host_wait_ms - wait0) / args.steps
    value = args.steps * (1 << log_n) * world / (elapsed_ms * 1e-3)

    # end to end through the C ABI: from the permutation inputs in pinned host memory (the trace
    # generated on the device), and from a whole witness in pinned host memory
    e2e = e2e_wit = None
    if not args.no_e2e:
        pin_in = torch.empty(16 << log_n, dtype=torch.int32, pin_memory=True)
        in_np = pin_in.numpy().view(np.uint32)
        in_np[:] = inputs

        def from_inputs():
            w = wl.Witness.generate(ctx, consts, in_np, log_n)
            try:
                return table.prove_witness(w)
            finally:
                w.free()

        for _ in range(max(1, args.warmup // 2)):
            from_inputs()
        barrier(world)
        torch.cuda.synchronize()
        e0.record(stream)
        for _ in range(args.steps):
            p1 = from_inputs()
        e1.record(stream)
        e1.synchronize()
        barrier(world)
        e2e_ms = dist_max(e0.elapsed_time(e1), world)
        assert np.array_equal(p1, proof)
        e2e = {"value": args.steps * (1 << log_n) * world / (e2e_ms * 1e-3), "unit": "perms/s",
               "h2d_bytes_per_step": int(in_np.nbytes), "d2h_bytes_per_step": int(p1.nbytes),
               "ms_per_step": e2e_ms / args.steps,
               "path": "inputs (16 per row) from pinned host memory, trace generated on the device "
                       "(wl_witness_generate, inside the timed region), wl_prove_witness, proof to the host"}

        host = torch.empty(165 << log_n, dtype=torch.int32, pin_memory=True)
        host_np = host.numpy().view(np.uint32)
        host_np[:] = wit.download()
        for _ in range(max(1, args.warmup // 2)):
            table.prove(host_np)
        barrier(world)
        torch.cuda.synchronize()
        e0.record(stream)
        for _ in range(args.steps):
            p2 = table.prove(host_np)
        e1.record(stream)
        e1.synchronize()
        barrier(world)
        e2e_ms = dist_max(e0.elapsed_time(e1), world)
        assert np.array_equal(p2, proof)
        e2e_wit = {"value": args.steps * (1 << log_n) * world / (e2e_ms * 1e-3), "unit": "perms/s",
                   "h2d_bytes_per_step": int(host_np.nbytes), "d2h_bytes_per_step": int(p2.nbytes),
                   "ms_per_step": e2e_ms / args.steps,
                   "path": "the whole witness from pinned host memory (wl_prove; the copy overlaps the "
                           "first commitment), proof to the host"}

    # the timed proof is checked by the library's host verifier (AirTable::verify), as the
    # reference verifies the proof it times (src/examples/poseidon2.rs:177-189)
    verified = wl.verify(consts, log_n, proof) == 0
    if rank != 0:
        return
    hbm_peak, hbm_source = read_hbm_peak()
    cpu = None
    if world == 1 and not args.no_cpu_baseline:
        cl = min(args.cpu_sample_log_n, log_n)
        rate, cores, sec = cpu_prove_rate(cl, 1, 0)
        cpu = {"value": rate, "unit": "perms/s", "cores": cores, "kind": "port",
               "sample": f"one CPU-oracle proof of 2^{cl} rows ({sec:.2f} s), all host threads",
               "cpu_model": cpu_model(), "nproc": os.cpu_count()}
    args.hbm_peak = hbm_peak
    batched = serving = sumcheck = None
    if world == 1 and not args.no_sumcheck:
        sumcheck = sumcheck_run(wl, ctx, args)
        if not args.no_cpu_baseline:
            sumcheck["cpu_baseline"] = sumcheck_cpu_baseline(args)
    if world == 1 and not args.no_batched:
        batched = batched_run(wl, args)
    if world == 1 and not args.no_serving:
        serving = serving_run(wl, args)
    line = {
        "metric": METRIC, "value": value, "unit": "perms/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": elapsed_ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "u32 (KoalaBear Montgomery; exact modular integer)",
        "data": "synthetic", "config": workload_config(log_n), "verified": bool(verified),
        "e2e": e2e, "e2e_host_witness": e2e_wit, "gpu_launches": launches, "clocks": clocks,
        "roofline": roofline(profile, breakdown, log_n, peaks, hbm_peak, args.steps, hbm_source),
        "cpu_baseline": cpu,
        "published_reference": {"value": 75000.0, "unit": "perms/s", "hardware": "Intel i9-12900H (CPU prover)",
                                "source": "reference README.md:20", "log_n_rows": 18},
        "int_peaks": peaks,
        "phases_ms": table.last_timings_ms,
        "host_syncs_per_step": host_syncs,
        "host_wait_ms_per_step": host_wait,
        "kernel_profile_ms": {k: round(v[0], 4) for k, v in sorted(breakdown.items(), key=lambda kv: -kv[1][0])},
        "kernel_profile_source": "CUDA events per kernel class over the last warm-up proof",
        "host_profile_ms": host_profile,
        "proof_len": int(proof.size),
        "autotune": wl.tune_report(),
        "sumcheck_microbench": sumcheck,
        "batched": batched,
        "serving": serving,
    }
    print(json.dumps(line), flush=True)


def main():
    args = parse_args()
    world, rank, local = dist_setup(args)
    if args.impl == "reference":
        run_reference(args, world, rank)
    else:
        run_ours(args, world, rank, local)
    if world > 1:
        import torch.distributed as dist
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
