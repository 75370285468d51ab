"""Benchmark of the B200 LDPC receive path.

One step = one batched decode of 8192 code blocks, BG1 / Zc=384
(A=8424, B=K=8448, N=25344), E=25344 LLRs per block (256QAM length,
rate 1/3), algo 1 (int16 layered min-sum, alpha=22936), 8 iterations, with
the rate recovery and per-iteration CRC check inside the kernel.

Inputs are synthetic int16 LLRs, round(128*LLR) clipped to +-10000 like the
reference channel model, drawn for random (non-codeword) bit sequences on a
BPSK/AWGN channel at Eb/N0 0.9 dB: the CRC never passes, so every one of the 8
iterations runs (the "noisy" case of the CPU baseline).  The inputs of one
step (415 MB) exceed the 126 MB L2, so no flush is needed between steps.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]

Prints one JSON line (rank 0).  N>1 runs one process per GPU under
torch.distributed.run (started here when no launcher did); every rank decodes
its own 8192 blocks (weak scaling, no collective on the data path; NCCL only
for the barrier and the max-time reduction).

Besides the timed step, the default single-GPU run adds, as extra keys of the
same line:
  * early_exit / config2_variants: device-encoded blocks through the 256QAM
    channel near the 1e-2 point (E=25344 algo 1, E=9600 algo 1, E=25344 BP);
  * parity: every block of the timed step and of those legs decoded again by
    the reference C decoder (oracle/_ref, one process per host core) and
    compared block by block; the same run gives cpu_baseline;
  * per_call: drop-in latency on the reference CUDA test's 8 cases;
  * mixed, serve, train: the mixed-size batch (every block checked against
    the reference), the serving loop and a training step, each with its own
    clock record (--no-legs skips them).
--impl reference times the reference C decoder alone on the GPU arm's own
blocks.
"""

from __future__ import annotations

import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import time

import numpy as np

REPO = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, REPO)

METRIC = "decoded info Gbit/s (BG1 Zc384 8it, bit-exact) vs CPU; serving p50/p99 TB latency"
CFG = (1, 8424, 1, 25344, 0, 8, 0)          # bgn, A, crctype, E, rv, Qm, HARQ_on
ROW = [1, 8, 22936, 0, 1280, 32767, -32767]  # algo 1, 8 iterations
N_CW = 8192
A_BITS = 8424
B_BITS = 8448
ZC = 384
NNZ = 316
E = 25344
EBN0_DB = 0.9
ESN0_1E2_DB = 11.0   # 256QAM Es/N0 of ~1e-2 BLER for this code, algo 1, 8 iterations (measured)
WORKLOAD = ("BG1 Zc=384 A=8424 B=8448 E=25344 (Qm=8 length, R=1/3), algo 1 int16 layered min-sum "
            "alpha=22936, 8 iterations (CRC never passes: all 8 run), 8192 code blocks per launch")


def algorithmic_bytes(iters: np.ndarray, E: int = E, fp: bool = False) -> float:
    """2E + ceil(B/8) + 4 + I_exec * (8*nnz*Zc + 2*B) per code block: every edge
    reads LQ and Lr and writes both (int16), plus the B hard-decision reads.
    Float decoders (algos 0, 4) move 4-byte values: I_exec * (16*nnz*Zc + 4*B)."""
    io = 2 * E + (B_BITS + 7) // 8 + 4
    per_it = (16 * NNZ * ZC + 4 * B_BITS) if fp else (8 * NNZ * ZC + 2 * B_BITS)
    return float(io * len(iters) + per_it * int(np.sum(iters)))


def synthetic_llrs(n: int, seed: int) -> np.ndarray:
    """n blocks of E int16 LLRs; every chunk of 256 blocks has its own generator
    (seed, chunk), so any process can regenerate any slice of the same blocks."""
    sigma = np.sqrt(0.5 / (10 ** (EBN0_DB / 10)))
    out = np.empty((n, E), dtype=np.int16)
    for s in range(0, n, 256):
        e = min(n, s + 256)
        rng = np.random.default_rng([seed, s // 256])
        x = 1.0 - 2.0 * rng.integers(0, 2, size=(e - s, E)).astype(np.float32)
        y = x + np.float32(sigma) * rng.standard_normal((e - s, E), dtype=np.float32)
        out[s:e] = np.clip(np.rint(y * np.float32(256.0 / sigma ** 2)), -10000, 10000).astype(np.int16)
    return out


def measured_peak():
    path = os.path.join(REPO, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


def _profile_constant(key):
    """A figure of the committed ncu summary of the decode kernel (`key: value`)."""
    path = os.path.join(REPO, "profiles", "fixed_pair_kernel_bg1_zc384.md")
    try:
        for line in open(path):
            if line.startswith(key + ":"):
                return float(line.split(":")[1].split()[0])
    except OSError:
        pass
    return None


def profiled_traffic():
    """DRAM bytes per code block of the decode kernel, from the committed ncu summary."""
    return _profile_constant("dram_bytes_per_codeword")


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled every 200 ms."""

    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self):
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None

    def stop(self):
        if not self.proc:
            return None
        self.proc.terminate()
        try:
            out, _ = self.proc.communicate(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
            out, _ = self.proc.communicate()
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in out.splitlines():
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                mx = max(mx, float(parts[2]))
            except ValueError:
                continue
            for name, val in zip(names, parts[5:9]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons), "samples": len(sm)}


# ----------------------------------------------------------------------------- reference decode of the same blocks
def _ref_check_worker(job):
    """Decode blocks [lo, hi) of `folder/llr.npy` on one host core with the
    reference C library built from its sources ("reference") or this repo's C
    restatement ("port"), timing only the decode calls, and compare every block
    with the GPU results saved beside the LLRs (when present)."""
    kind, folder, lo, hi, cfg_t, row = job
    sys.path.insert(0, REPO)
    from oracle.oracle import Oracle, RefLib, dec_cfg, in_config

    cfg, dcfg = in_config(*cfg_t), dec_cfg(row)
    fp = row[0] in (0, 4)
    llr = np.load(os.path.join(folder, "llr.npy"), mmap_mode="r")
    gpu = None
    if os.path.exists(os.path.join(folder, "status.npy")):
        gpu = {k: np.load(os.path.join(folder, k + ".npy"), mmap_mode="r")
               for k in ("status", "hardbits", "iterations", "app")}
    if kind == "reference":
        ref = RefLib()
        rc, p = ref.gen(cfg)
        acc = {1: ref.lib.ref_fixed_lq, 2: ref.lib.ref_neural_lq, 3: ref.lib.ref_degree_lq,
               0: ref.lib.ref_float_lq, 4: ref.lib.ref_float_lq}[row[0]]
        fn = ref.lib.c_ldpc_5g_decode
    else:
        orc = Oracle()
        rc, p = orc.derive(cfg)
    assert rc == 0
    n_app = p.N + 2 * p.Zc
    nb = (p.B + 7) // 8
    bits = np.zeros(nb, dtype=np.uint8)
    lq = np.zeros(n_app, dtype=np.float32 if fp else np.int16)
    it = ctypes.c_int32(0)
    r = {"t": 0.0, "n": hi - lo, "converged": 0, "status": 0, "hardbits_blocks": 0, "hardbits_bits": 0,
         "iterations": 0, "iterations_compared": 0, "app_blocks": 0, "llr_beyond_1e-4": 0, "llr_sign": 0,
         "llr_max_abs": 0.0, "llr_values": 0}
    for i in range(lo, hi):
        x = np.ascontiguousarray(llr[i], dtype=np.int16)
        bits[:] = 0
        if kind == "reference":
            t0 = time.perf_counter()
            st = fn(x.ctypes.data, bits.ctypes.data, ctypes.byref(cfg), ctypes.byref(dcfg))
            r["t"] += time.perf_counter() - t0
            lq = np.ctypeslib.as_array(acc(), shape=(n_app,))
            its = row[1] if st == 1 else None      # the reference does not report its iteration count
        else:
            t0 = time.perf_counter()
            st = orc.lib.orc_decode(x.ctypes.data, bits.ctypes.data, ctypes.byref(cfg), ctypes.byref(dcfg),
                                    orc.harq.ctypes.data, lq.ctypes.data, ctypes.byref(it))
            r["t"] += time.perf_counter() - t0
            its = int(it.value)
        r["converged"] += int(st == 0)
        if gpu is None:
            continue
        r["status"] += int(int(gpu["status"][i]) != st)
        diff = int(np.unpackbits(np.bitwise_xor(np.asarray(gpu["hardbits"][i][:nb]), bits)).sum())
        r["hardbits_blocks"] += int(diff > 0)
        r["hardbits_bits"] += diff
        if its is not None:
            r["iterations_compared"] += 1
            r["iterations"] += int(int(gpu["iterations"][i]) != its)
        g = np.asarray(gpu["app"][i][:n_app])
        if fp:
            d = np.abs(g.astype(np.float64) - lq.astype(np.float64))
            r["llr_values"] += n_app
            r["llr_beyond_1e-4"] += int(np.sum(d > 1e-4 * np.abs(lq) + 1e-6))
            r["llr_sign"] += int(np.sum(np.signbit(g) != np.signbit(lq)))
            r["llr_max_abs"] = max(r["llr_max_abs"], float(d.max()))
            r["app_blocks"] += int(not np.array_equal(g, lq))
        else:
            r["app_blocks"] += int(not np.array_equal(g, lq))
    return r


def reference_decode(host_llr, cfg, row, gpu=None, procs: int = 0, a_bits: int = A_BITS) -> dict:
    """Decode every block of `host_llr` with the reference C decoder (built from
    its sources into oracle/_ref; else the oracle port) in one process per host
    core (the reference decoders keep state in file-static buffers), timing the
    decode calls.  With `gpu` (numpy status, hardbits, iterations, app of the
    same blocks) every block is compared field by field."""
    import multiprocessing as mp
    import shutil
    import tempfile

    from oracle.oracle import REF_SO

    kind = "reference" if os.path.exists(REF_SO) else "port"
    n = host_llr.shape[0]
    procs = max(1, min(procs or len(os.sched_getaffinity(0)) or 1, n))
    folder = tempfile.mkdtemp(prefix="ldpc_refcheck_")
    try:
        np.save(os.path.join(folder, "llr.npy"), host_llr)
        if gpu is not None:
            for k in ("status", "hardbits", "iterations", "app"):
                np.save(os.path.join(folder, k + ".npy"), gpu[k])
        bounds = [(r * n // procs, (r + 1) * n // procs) for r in range(procs)]
        jobs = [(kind, folder, lo, hi, tuple(cfg), list(row)) for lo, hi in bounds]
        t0 = time.perf_counter()
        with mp.get_context("spawn").Pool(procs) as pool:
            parts = pool.map(_ref_check_worker, jobs)
        wall = time.perf_counter() - t0
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    slowest = max(p["t"] for p in parts)
    tot = {k: sum(p[k] for p in parts) for k in parts[0] if k not in ("t", "llr_max_abs")}
    out = {"kind": kind, "cores": procs, "blocks": n, "slowest_s": slowest, "wall_s": wall,
           "gbps": n * a_bits / slowest / 1e9, "converged": tot["converged"]}
    if gpu is not None:
        fp = row[0] in (0, 4)
        par = {"blocks": n, "against": ("reference c_lib built from its sources (oracle/_ref), c_ldpc_5g_decode"
                                        if kind == "reference" else "C restatement of the reference (oracle port)"),
               "status_mismatches": tot["status"], "hardbit_block_mismatches": tot["hardbits_blocks"],
               "hardbit_mismatches": tot["hardbits_bits"],
               "iteration_mismatches": tot["iterations"], "iterations_compared": tot["iterations_compared"],
               "final_llr_block_mismatches": tot["app_blocks"]}
        if fp:
            par.update({"llr_values": tot["llr_values"], "llr_beyond_1e-4_rel": tot["llr_beyond_1e-4"],
                        "llr_beyond_1e-4_rate": tot["llr_beyond_1e-4"] / max(1, tot["llr_values"]),
                        "llr_sign_mismatches": tot["llr_sign"],
                        "llr_max_abs_diff": max(p["llr_max_abs"] for p in parts),
                        "hardbit_block_mismatch_rate": tot["hardbits_blocks"] / n})
            par["mismatches"] = tot["status"] + tot["hardbits_blocks"] + tot["iterations"]
            par["fields"] = "status, hard bits, iterations (exact); final float LLRs (statistics)"
        else:
            par["mismatches"] = tot["status"] + tot["hardbits_blocks"] + tot["iterations"] + tot["app_blocks"]
            par["fields"] = "status, hard bits, iterations, final int16 LLRs (all exact)"
        if kind == "reference":
            par["iterations_note"] = ("the reference reports no iteration count: compared where it is implied "
                                      "(status 1 = max_iterations); the final LLRs pin the exit iteration")
        out["parity"] = par
    return out


def _ref_mixed_worker(job):
    """Blocks [lo, hi) of a mixed-size batch: each decoded alone by the
    reference C library (status, hard bits) and by the oracle port (which also
    reports the iteration count), and compared with the GPU's results."""
    folder, lo, hi, row = job
    sys.path.insert(0, REPO)
    from oracle.oracle import REF_SO, Oracle, RefLib, dec_cfg, in_config

    cfgs = np.load(os.path.join(folder, "cfgs.npy"))            # [n, 8]: bgn, A, crc, E, rv, Qm, llr_off, bits_off
    arena = np.load(os.path.join(folder, "llr.npy"), mmap_mode="r")
    g_bits = np.load(os.path.join(folder, "bits.npy"), mmap_mode="r")
    g_st = np.load(os.path.join(folder, "status.npy"))
    g_it = np.load(os.path.join(folder, "iterations.npy"))
    ref = RefLib() if os.path.exists(REF_SO) else None
    orc = Oracle()
    dcfg = dec_cfg(row)
    r = {"n": hi - lo, "ref_status": 0, "ref_bits": 0, "orc_status": 0, "orc_bits": 0, "orc_iters": 0, "converged": 0}
    for i in range(lo, hi):
        bgn, A, crc, E, rv, Qm, lo_off, bo = (int(v) for v in cfgs[i])
        cfg = in_config(bgn, A, crc, E, rv, Qm, 0)
        x = np.ascontiguousarray(arena[lo_off:lo_off + E], dtype=np.int16)
        st, bits, it, _ = orc.decode(x, cfg, dcfg)
        nb = len(bits)
        got = np.asarray(g_bits[bo:bo + nb])
        r["converged"] += int(st == 0)
        r["orc_status"] += int(st != int(g_st[i]))
        r["orc_iters"] += int(it != int(g_it[i]))
        r["orc_bits"] += int(it > 0 and not np.array_equal(got, bits))
        if ref is not None:
            rst, rbits, _ = ref.decode(x, cfg, dcfg)
            r["ref_status"] += int(rst != int(g_st[i]))
            r["ref_bits"] += int(it > 0 and not np.array_equal(got, rbits[:nb]))
    return r


def reference_decode_mixed(arena_h, cfgs, llr_offs, bits_offs, gpu_bits, gpu_status, gpu_iters, row, procs=0):
    """Every block of a mixed-size batch decoded alone on the host cores and
    compared with the GPU's results of the batch."""
    import multiprocessing as mp
    import shutil
    import tempfile

    from oracle.oracle import REF_SO

    n = len(cfgs)
    procs = max(1, min(procs or len(os.sched_getaffinity(0)) or 1, n))
    folder = tempfile.mkdtemp(prefix="ldpc_mixedcheck_")
    try:
        tab = np.array([list(c) + [lo, bo] for c, lo, bo in zip(cfgs, llr_offs, bits_offs)], dtype=np.int64)
        np.save(os.path.join(folder, "cfgs.npy"), tab)
        np.save(os.path.join(folder, "llr.npy"), arena_h)
        np.save(os.path.join(folder, "bits.npy"), gpu_bits)
        np.save(os.path.join(folder, "status.npy"), gpu_status)
        np.save(os.path.join(folder, "iterations.npy"), gpu_iters)
        jobs = [(folder, k * n // procs, (k + 1) * n // procs, list(row)) for k in range(procs)]
        t0 = time.perf_counter()
        with mp.get_context("spawn").Pool(procs) as pool:
            parts = pool.map(_ref_mixed_worker, jobs)
        wall = time.perf_counter() - t0
    finally:
        shutil.rmtree(folder, ignore_errors=True)
    tot = {k: sum(p[k] for p in parts) for k in parts[0]}
    against = ("reference c_lib built from its sources (status, hard bits) and the oracle port (status, hard bits, "
               "iterations), each block decoded alone" if os.path.exists(REF_SO) else
               "the oracle port (status, hard bits, iterations), each block decoded alone")
    return {"blocks": n, "against": against,
            "reference_status_mismatches": tot["ref_status"], "reference_hardbit_mismatches": tot["ref_bits"],
            "oracle_status_mismatches": tot["orc_status"], "oracle_hardbit_mismatches": tot["orc_bits"],
            "oracle_iteration_mismatches": tot["orc_iters"],
            "mismatches": tot["ref_status"] + tot["ref_bits"] + tot["orc_status"] + tot["orc_bits"] + tot["orc_iters"],
            "converged": tot["converged"], "cores": procs, "wall_s": round(wall, 1)}


def cpu_baseline_from(ref: dict, what: str) -> dict:
    return {"value": ref["gbps"], "unit": "Gbit/s", "cores": ref["cores"], "kind": ref["kind"],
            "sample": (f"{what}: {ref['blocks']} code blocks split over {ref['cores']} processes (one per host "
                       f"core), sum of A bits / slowest process's decode time ({ref['slowest_s']:.1f} s; "
                       f"pool wall {ref['wall_s']:.1f} s)")}


def gpu_results(res, n_app=None) -> dict:
    """Host copies of a DecodeResult for the reference comparison."""
    return {"status": res.status.cpu().numpy(), "hardbits": res.hardbits.cpu().numpy(),
            "iterations": res.iterations.cpu().numpy(), "app": res.app.cpu().numpy()}


# ----------------------------------------------------------------------------- GPU arm
def run_gpu(args, rank, world, local_rank):
    import torch

    from deeplearning_5g_ldpc_decoder_b200.shard import max_over_ranks, sum_over_ranks

    from deeplearning_5g_ldpc_decoder_b200 import capi, ldpc_decode

    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist

        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120), device_id=dev)

    n_cw = args.n_cw
    host_llr = synthetic_llrs(n_cw, seed=rank)
    d_llr = torch.from_numpy(host_llr).to(dev)
    lib = capi.load_library()
    out = None
    stream = torch.cuda.current_stream(dev)

    def barrier():
        if dist is not None:
            dist.barrier()
        torch.cuda.synchronize(dev)

    # ---- kernel-resident timing (inputs already in HBM) ----
    row = list(ROW)
    row[0] = args.algo
    for _ in range(max(args.warmup, 0)):
        out = ldpc_decode(d_llr, CFG, row, out=out)
    barrier()
    launches0 = capi.kernel_launch_count()
    sampler = ClockSampler() if rank == 0 else None
    if sampler:
        sampler.start()
        time.sleep(0.3)
    ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(args.steps)]
    barrier()
    t_start = torch.cuda.Event(enable_timing=True)
    t_end = torch.cuda.Event(enable_timing=True)
    t_start.record(stream)
    for k in range(args.steps):
        ev[k][0].record(stream)
        out = ldpc_decode(d_llr, CFG, row, out=out)
        ev[k][1].record(stream)
    t_end.record(stream)
    barrier()
    clocks = sampler.stop() if sampler else None
    launches = capi.kernel_launch_count() - launches0
    total_ms = t_start.elapsed_time(t_end)
    launch_ms = [a.elapsed_time(b) for a, b in ev]
    iters = out.iterations.cpu().numpy()
    status = out.status.cpu().numpy()
    ms_step = max_over_ranks(total_ms / args.steps, dist, dev)
    info_bits = sum_over_ranks(n_cw * A_BITS, dist, dev)
    # the blocks of the timed step once more with their final beliefs (untimed), for the reference comparison
    checks = []
    do_parity = rank == 0 and world == 1 and not args.no_parity
    if do_parity:
        chk = ldpc_decode(d_llr, CFG, row, return_app=True)
        torch.cuda.synchronize(dev)
        assert torch.equal(chk.hardbits, out.hardbits) and torch.equal(chk.status, out.status) \
            and torch.equal(chk.iterations, out.iterations), "the final-belief launch differs from the timed one"
        checks.append(("main", host_llr, CFG, row, gpu_results(chk)))
        del chk

    # ---- realistic inputs: device-encoded code blocks through the 256QAM channel
    # near the 1e-2 BLER point; CRC early termination as in the reference ----
    early = None
    variants = None
    if not args.no_e2e:
        early = run_early_exit(args, n_cw, dev, stream, barrier, dist, torch, checks=checks if do_parity else None)
        variants = run_config2_variants(args, n_cw, dev, stream, barrier, dist, torch,
                                        checks=checks if do_parity else None)

    # ---- end to end through the host-buffer C ABI (pinned memory) ----
    if args.no_e2e:
        e2e_ms = float("nan")
    else:
        e2e_ms = run_e2e(args, lib, host_llr, out, stream, barrier, dist, dev, iters, torch)

    per_call = run_per_call(args) if (rank == 0 and world == 1 and not args.no_e2e) else None

    # ---- every block of every leg decoded again by the reference C decoder on the host cores ----
    refs = {}
    for name, llr_h, cfg, row_c, gpu in checks:
        refs[name] = reference_decode(llr_h, cfg, row_c, gpu=gpu, procs=args.cpu_procs,
                                      a_bits=cfg[1])
    result = None
    if rank == 0:
        value = info_bits / (ms_step * 1e-3) / 1e9
        e2e_value = info_bits / (e2e_ms * 1e-3) / 1e9
        alg = algorithmic_bytes(iters, fp=args.algo in (0, 4))
        mean_launch_ms = float(np.mean(launch_ms))
        achieved = alg / (mean_launch_ms * 1e-3) / 1e9
        peak, peak_kind = measured_peak()
        traffic_cw = profiled_traffic() if args.algo == 1 else None
        nb = (B_BITS + 7) // 8
        result = {
            "metric": METRIC,
            "value": round(value, 4),
            "unit": "Gbit/s",
            "n_gpus": world,
            "steps": args.steps,
            "warmup": args.warmup,
            "ms_per_step": round(ms_step, 4),
            "higher_is_better": True,
            "scaling": "weak",
            "vs_baseline": None,
            "dtype": "f32" if args.algo in (0, 4) else "int16",
            "data": "synthetic: seeded int16 LLRs (round(128*LLR), +-10000 clip) of random bits on BPSK/AWGN at "
                    "Eb/N0 0.9 dB; CRC never passes so all 8 iterations run",
            "config": {"workload": WORKLOAD.replace("8192", str(n_cw)).replace(
                           "algo 1 int16 layered min-sum alpha=22936",
                           {0: "algo 0 float BP", 1: "algo 1 int16 layered min-sum alpha=22936",
                            2: "algo 2 int16 trained-table min-sum", 3: "algo 3 int16 degree min-sum",
                            4: "algo 4 float min-sum alpha=22936"}[args.algo]),
                       "code_blocks_per_step_per_gpu": n_cw,
                       "parallelism": f"replicas x{world}, independent code blocks per GPU",
                       "l2": f"inputs {n_cw * E * 2 / 1e6:.0f} MB per step vs 126 MB L2"},
            "e2e": {"value": round(e2e_value, 4), "unit": "Gbit/s",
                    "h2d_bytes_per_step": int(n_cw * E * 2),
                    "d2h_bytes_per_step": int(n_cw * (nb + 8)),
                    "path": "nrldpc_decode_batch_host (C ABI) from pinned host buffers, copies in the timed region",
                    "ms_per_step": round(e2e_ms, 4)},
            "roofline": {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
                         "frac": round(achieved / peak, 4), "peak_kind": f"{peak_kind} (MEASURED_PEAKS.json hbm_gbs)",
                         "traffic": (round(traffic_cw * n_cw) if traffic_cw else None),
                         "traffic_source": ("profile constant, not measured in this run: ncu dram__bytes_read.sum + "
                                            "dram__bytes_write.sum per block of the committed capture "
                                            "(profiles/fixed_pair_kernel_bg1_zc384.md) x blocks per launch"
                                            if traffic_cw else "no ncu capture of this decoder's launch"),
                         "algorithmic_bytes_per_launch": alg, "kernel_ms": round(mean_launch_ms, 4),
                         "note": ("the algorithmic bytes count every belief and message access as HBM traffic; "
                                  "this decoder keeps beliefs in shared memory and messages mostly in L2, "
                                  "so it runs above that model, and what limits it is the "
                                  "integer ALU pipe (profile constant alu_pipe_busy)") if args.algo == 1 else None,
                         "alu_pipe_busy": _profile_constant("alu_pipe_busy") if args.algo == 1 else None,
                         "io_bytes_per_launch": float((2 * E + (B_BITS + 7) // 8 + 4) * n_cw)},
            "iterations_executed_mean": float(np.mean(iters)),
            "converged": int(np.sum(status == 0)),
            "early_exit": early,
            "config2_variants": variants,
            "per_call": per_call,
            "gpu_launches": int(launches),
            "clocks": clocks,
        }
        if "main" in refs:
            result["parity"] = refs["main"]["parity"]
            result["cpu_baseline"] = cpu_baseline_from(
                refs["main"], "the timed step's own blocks (seed 0, noisy, all 8 iterations run)")
        for leg in (early, *(variants or {}).values()):
            if leg is not None and leg.get("_check") in refs:
                ref = refs[leg.pop("_check")]
                leg["parity"] = ref["parity"]
                leg["reference_cpu_gbps"] = round(ref["gbps"], 6)
                leg["reference_converged"] = ref["converged"]
        if args.no_e2e:
            result["e2e"] = None
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    return result


def _esn0_for_bler(cfg, row, Qm, target, dev, torch, n_cw: int = 2048, lo: float = 0.0, hi: float = 35.0):
    """Es/N0 (dB) where the block error rate of device-encoded blocks through the
    device channel crosses `target` (bisection, 10 steps)."""
    from deeplearning_5g_ldpc_decoder_b200 import channel_llrs, ldpc_decode, ldpc_encode

    gen = torch.Generator(device=dev).manual_seed(77)
    pay = torch.randint(0, 256, (n_cw, cfg[1] // 8), dtype=torch.uint8, device=dev, generator=gen)
    rm = ldpc_encode(pay, cfg)
    for k in range(10):
        mid = 0.5 * (lo + hi)
        res = ldpc_decode(channel_llrs(rm, cfg[3], Qm, -mid, seed=500 + k), cfg, row)
        ok = (res.status == 0) & (res.hardbits[:, : cfg[1] // 8] == pay).all(dim=1)
        if 1.0 - float(ok.float().mean()) > target:
            lo = mid
        else:
            hi = mid
    return round(0.5 * (lo + hi), 2)


def run_early_exit(args, n_cw, dev, stream, barrier, dist, torch, cfg=None, row=None, esn0=None, checks=None,
                   name="early_exit"):
    """Realistic inputs: device-encoded payloads through the 256QAM channel at the
    given Es/N0, CRC early termination as in the reference.  With `checks`, the
    leg's LLRs and final beliefs are queued for the reference comparison."""
    from deeplearning_5g_ldpc_decoder_b200.shard import max_over_ranks
    from deeplearning_5g_ldpc_decoder_b200 import channel_llrs, ldpc_decode, ldpc_encode

    cfg = cfg or CFG
    row = row or ROW
    esn0 = ESN0_1E2_DB if esn0 is None else esn0
    gen = torch.Generator(device=dev).manual_seed(1234)
    pay = torch.randint(0, 256, (n_cw, A_BITS // 8), dtype=torch.uint8, device=dev, generator=gen)
    llr = channel_llrs(ldpc_encode(pay, cfg), cfg[3], 8, noise_power_db=-esn0, seed=99)
    out = None
    for _ in range(max(args.warmup, 1)):
        out = ldpc_decode(llr, cfg, row, out=out)
    barrier()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        out = ldpc_decode(llr, cfg, row, out=out)
    e1.record(stream)
    barrier()
    ms = max_over_ranks(e0.elapsed_time(e1) / args.steps, dist, dev)
    ok = (out.status == 0) & (out.hardbits[:, : A_BITS // 8] == pay).all(dim=1)
    iters = out.iterations.cpu().numpy()
    world = dist.get_world_size() if dist is not None else 1
    fp = row[0] in (0, 4)
    leg = {"value": round(n_cw * A_BITS * world / (ms * 1e-3) / 1e9, 4), "unit": "Gbit/s", "ms_per_step": round(ms, 4),
           "iterations_executed_mean": float(np.mean(iters)), "bler": float(1.0 - ok.float().mean().item()),
           "roofline_achieved_gbs": round(algorithmic_bytes(iters, E=cfg[3], fp=fp) / (ms * 1e-3) / 1e9, 1),
           "inputs": f"device-encoded random payloads, E={cfg[3]}, 256QAM AWGN at Es/N0 {esn0} dB, max-log LLRs "
                     "quantised like the reference channel",
           "decoder": {0: "algo 0 float BP", 1: "algo 1 int16 min-sum", 4: "algo 4 float min-sum"}.get(row[0], str(row[0]))}
    if checks is not None:
        chk = ldpc_decode(llr, cfg, row, return_app=True)
        torch.cuda.synchronize(dev)
        assert torch.equal(chk.hardbits, out.hardbits) and torch.equal(chk.status, out.status)
        checks.append((name, llr.cpu().numpy(), cfg, row, gpu_results(chk)))
        leg["_check"] = name
        del chk
    return leg


def run_config2_variants(args, n_cw, dev, stream, barrier, dist, torch, checks=None):
    """The other legs of the large single-size batch: E=9600 (rate 0.88) with algo 1,
    and algo 0 (float BP) at E=25344, each at its measured ~1e-2 BLER point."""
    cfg88 = (1, 8424, 1, 9600, 0, 8, 0)
    row_bp = [0, 8, 22936, 0, 1280, 32767, -32767]
    esn0_88 = _esn0_for_bler(cfg88, ROW, 8, 0.01, dev, torch)
    esn0_bp = _esn0_for_bler(CFG, row_bp, 8, 0.01, dev, torch, n_cw=1024, lo=5.0, hi=15.0)
    out = {"E9600_algo1": run_early_exit(args, n_cw, dev, stream, barrier, dist, torch, cfg88, ROW, esn0_88,
                                         checks=checks, name="E9600_algo1"),
           "E25344_algo0_bp": run_early_exit(args, n_cw, dev, stream, barrier, dist, torch, CFG, row_bp, esn0_bp,
                                             checks=checks, name="E25344_algo0_bp")}
    return out


def run_e2e(args, lib, host_llr, out, stream, barrier, dist, dev, iters, torch):
    from deeplearning_5g_ldpc_decoder_b200.shard import max_over_ranks
    from deeplearning_5g_ldpc_decoder_b200.capi import make_decoder_config, make_in_config

    n_cw = host_llr.shape[0]
    pin_llr = torch.from_numpy(host_llr).pin_memory()
    nb = (B_BITS + 7) // 8
    pin_bits = torch.zeros((n_cw, nb), dtype=torch.uint8).pin_memory()
    pin_stat = torch.zeros(n_cw, dtype=torch.int32).pin_memory()
    pin_it = torch.zeros(n_cw, dtype=torch.int32).pin_memory()
    icfg, dcfg = make_in_config(*CFG), make_decoder_config(ROW)
    sptr = ctypes.c_void_p(stream.cuda_stream)

    def e2e_step():
        rc = lib.nrldpc_decode_batch_host(
            ctypes.c_void_p(pin_llr.data_ptr()), E, n_cw, ctypes.byref(icfg), ctypes.byref(dcfg),
            ctypes.c_void_p(pin_bits.data_ptr()), nb, ctypes.c_void_p(pin_stat.data_ptr()),
            ctypes.c_void_p(pin_it.data_ptr()), sptr)
        if rc != 0:
            raise RuntimeError(f"nrldpc_decode_batch_host failed: {rc}")

    for _ in range(max(args.warmup, 1)):
        e2e_step()
    barrier()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(args.steps):
        e2e_step()
    e1.record(stream)
    barrier()
    e2e_ms = max_over_ranks(e0.elapsed_time(e1) / args.steps, dist, dev)
    assert np.array_equal(pin_it.numpy(), iters) and np.array_equal(pin_bits.numpy(), out.hardbits.cpu().numpy())

    return e2e_ms


PER_CALL_CASES = [(1, 488, 1, 1536, 0, 1, 0), (1, 1024, 0, 3072, 0, 1, 0), (1, 2400, 2, 8192, 0, 1, 0),
                  (1, 4072, 1, 16384, 0, 1, 0), (2, 176, 1, 512, 0, 1, 0), (2, 640, 3, 2048, 0, 1, 0),
                  (2, 1200, 0, 4096, 0, 1, 0), (2, 2400, 2, 8192, 0, 1, 0)]
PER_CALL_ROW = [1, 32, 22936, 0, 1280, 32767, -32767]


def run_per_call(args, warmup: int = 2, calls: int = 20) -> dict:
    """Latency of one drop-in call (cuda_ldpc_5g_decode with host buffers: copy in,
    decode, copy out, return) on the 8 cases and with the protocol of the
    reference's CUDA decoder test (CUDA/test_ldpc_5g_decoder.cu:318-327: BPSK at
    0 dB, algo 1, 32 iterations; :271-309: 2 warm-up then 20 timed calls, the
    hard-bit buffer cleared before each).  Inputs come from this library's own
    encoder and channel (cuda_ldpc_5g_encode, tx_rx_process).  The reference C
    decoder, timed on the same LLRs by the same protocol on one host core, is
    the CPU side; hard bits and status must agree."""
    from deeplearning_5g_ldpc_decoder_b200 import capi

    lib = capi.load_library()
    ref = None
    if not args.no_parity:
        from oracle.oracle import REF_SO, RefLib

        if os.path.exists(REF_SO):
            ref = RefLib()
    dcfg = capi.make_decoder_config(PER_CALL_ROW)
    rng = np.random.default_rng(2000)
    cases = []
    for k, c in enumerate(PER_CALL_CASES):
        icfg = capi.make_in_config(*c)
        p = capi.gen_ldpc_parameters(icfg)
        info = np.zeros(1056, dtype=np.uint8)
        info[: c[1] // 8] = rng.integers(0, 256, c[1] // 8, dtype=np.uint8)
        rm = np.zeros((c[3] + 7) // 8 + 8, dtype=np.uint8)
        assert lib.cuda_ldpc_5g_encode(info.ctypes.data, rm.ctypes.data, ctypes.byref(icfg)) == 0
        lib.nrldpc_channel_seed(1000 + c[1] + c[3] + c[5] * 17)
        llr = np.zeros(c[3], dtype=np.int16)
        assert lib.tx_rx_process(rm.ctypes.data, c[3], c[5], ctypes.c_float(0.0), llr.ctypes.data) == 0
        nb = (p.B + 7) // 8
        bits = np.zeros(nb, dtype=np.uint8)

        def timed(fn, ic, dc):
            for _ in range(warmup):
                bits[:] = 0
                st = fn(llr.ctypes.data, bits.ctypes.data, ctypes.byref(ic), ctypes.byref(dc))
            t0 = time.perf_counter()
            for _ in range(calls):
                bits[:] = 0
                st = fn(llr.ctypes.data, bits.ctypes.data, ctypes.byref(ic), ctypes.byref(dc))
            return (time.perf_counter() - t0) * 1e3 / calls, int(st), bits.copy()

        ms, st, got = timed(lib.cuda_ldpc_5g_decode, icfg, dcfg)
        ok = st == 0 and np.array_equal(got[: c[1] // 8], info[: c[1] // 8])
        leg = {"case": list(c), "Zc": int(p.Zc), "ms_per_call": round(ms, 4), "status": st, "payload_ok": bool(ok)}
        if ref is not None:
            from oracle.oracle import dec_cfg, in_config

            rms, rst, rbits = timed(ref.lib.c_ldpc_5g_decode, in_config(*c), dec_cfg(PER_CALL_ROW))
            leg.update({"reference_c_ms_per_call": round(rms, 4), "reference_status": rst,
                        "same_result": bool(rst == st and np.array_equal(rbits, got)),
                        "speedup": round(rms / ms, 2)})
        cases.append(leg)
    head = cases[3]
    return {"protocol": f"{warmup} warm-up + {calls} timed calls per case, host buffers, synchronous return "
                        "(CUDA/test_ldpc_5g_decoder.cu:271-309); BPSK at 0 dB, algo 1, 32 iterations",
            "headline_case": "cases[3] = (1, 4072, 1, 16384, 0, 1, 0), the case the reference test profiles",
            "ms_per_call": head["ms_per_call"], "reference_c_ms_per_call": head.get("reference_c_ms_per_call"),
            "cases": cases}


def run_mixed(args):
    """Mixed-size batch: one persistent kernel under a CUDA graph vs one plain
    launch per block through the uniform entry point, same inputs."""
    import torch

    from deeplearning_5g_ldpc_decoder_b200 import capi, channel_llrs, ldpc_decode, ldpc_encode
    from deeplearning_5g_ldpc_decoder_b200.mixed import AUTOTUNE_NAMES, MixedPlan, random_mixed_configs

    n = args.n_cw if args.n_cw != N_CW else 32768
    row = [1, 10, 22936, 0, 1280, 32767, -32767]
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    # first transmissions (rv 0): a lone rv 1-3 block can lack systematic bits
    cfgs = random_mixed_configs(n, seed=2024, rvs=(0,))
    gen = torch.Generator(device=dev).manual_seed(7)
    llrs, pays = [], []
    for i, (bgn, A, crc, E, rv, Qm) in enumerate(cfgs):
        pay = torch.randint(0, 256, (1, max(A // 8, 1)), dtype=torch.uint8, device=dev, generator=gen)[:, : A // 8]
        rm = ldpc_encode(pay.contiguous(), (bgn, A, crc, E, rv, Qm, 0))
        # Es/N0 = Shannon bound of the block's spectral efficiency + 3.5 dB, spread by 0..2 dB
        # (max-log QAM + 10 min-sum iterations need ~2-4 dB above the bound: block error rate ~10 %)
        eta = (A + 24) / E * Qm
        snr = 10.0 * np.log10(2.0 ** eta - 1.0) + 3.5 + 0.5 * (i % 5)
        llrs.append(channel_llrs(rm, E, Qm, -snr, seed=i)[0])
        pays.append(pay[0])
    plan = MixedPlan(cfgs, row, device=dev)
    arena = torch.cat(llrs)
    stream = torch.cuda.Stream(dev)
    with torch.cuda.stream(stream):
        out = plan.outputs()
        best, cand_ms = plan.autotune(arena, out=out)
        for _ in range(max(args.warmup, 1)):
            plan.decode(arena, use_graph=True, out=out)
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        launches0 = capi.kernel_launch_count()
        e0.record(stream)
        for _ in range(args.steps):
            plan.decode(arena, use_graph=True, out=out)
        e1.record(stream)
    stream.synchronize()
    ms_mixed = e0.elapsed_time(e1) / args.steps
    launches = capi.kernel_launch_count() - launches0
    bits, status, iters = out
    st = status.cpu().numpy()
    b = bits.cpu().numpy()
    ok = np.array([st[i] == 0 and np.array_equal(b[plan.bits_offsets[i]: plan.bits_offsets[i] + len(pays[i])],
                                                 pays[i].cpu().numpy()) for i in range(n)])
    # plain per-block launches of the uniform entry point (C ABI, preallocated outputs)
    lib = capi.load_library()
    dcfg = capi.make_decoder_config(row)
    icfgs = [capi.make_in_config(*c, 0) for c in cfgs]
    pbits = torch.zeros((n, 1056), dtype=torch.uint8, device=dev)
    pst = torch.empty(n, dtype=torch.int32, device=dev)
    pit = torch.empty(n, dtype=torch.int32, device=dev)
    sptr = ctypes.c_void_p(stream.cuda_stream)
    args_i = [(ctypes.c_void_p(llrs[i].data_ptr()), cfgs[i][3], 1, ctypes.byref(icfgs[i]), ctypes.byref(dcfg),
               ctypes.c_void_p(pbits[i].data_ptr()), 1056, ctypes.c_void_p(pst[i:].data_ptr()),
               ctypes.c_void_p(pit[i:].data_ptr()), ctypes.c_void_p(0), 0, ctypes.c_void_p(0), 0, sptr)
              for i in range(n)]
    for i in range(min(64, n)):
        lib.nrldpc_decode_batch(*args_i[i])
    e0.record(stream)
    for i in range(n):
        lib.nrldpc_decode_batch(*args_i[i])
    e1.record(stream)
    stream.synchronize()
    ms_plain = e0.elapsed_time(e1)
    assert torch.equal(pst.cpu(), status.cpu())
    info = sum(c[1] for c in cfgs)
    parity = None
    if not args.no_parity:
        parity = reference_decode_mixed(arena.cpu().numpy(), cfgs, plan.llr_offsets, plan.bits_offsets, b, st,
                                        iters.cpu().numpy(), row, procs=args.cpu_procs)
    return {"metric": METRIC, "value": round(info / (ms_mixed * 1e-3) / 1e9, 4), "unit": "Gbit/s", "n_gpus": 1,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms_mixed, 4), "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "int16",
            "data": "synthetic: device-encoded random payloads through the device QAM/AWGN channel, Es/N0 spread",
            "config": {"workload": f"mixed: {n} blocks, Zc uniform over 51 sizes, BG1 60 %, rate U[0.2,0.92], "
                                   "Qm {2,4,6,8}, rv 0, CRC24 type random, algo 1, 10 iterations, CRC early exit",
                       "parallelism": "single GPU, one persistent kernel, CUDA graph replay"},
            "plain_per_block_launches": {"value": round(info / (ms_plain * 1e-3) / 1e9, 4), "unit": "Gbit/s",
                                         "ms_per_step": round(ms_plain, 3), "launches": n,
                                         "path": "nrldpc_decode_batch once per block (C ABI), same inputs"},
            "speedup_vs_plain": round(ms_plain / ms_mixed, 2),
            "autotune": {"chosen": best, "candidates_ms": [round(x, 4) for x in cand_ms],
                         "candidates": AUTOTUNE_NAMES},
            "iterations_executed_mean": float(iters.float().mean().item()), "bler": float(1.0 - ok.mean()),
            "parity": parity, "gpu_launches": int(launches)}


SERVE_MCS = [(2, 0.30), (2, 0.60), (4, 0.45), (4, 0.70), (6, 0.55), (6, 0.75), (8, 0.70), (8, 0.85)]


def _cb_error_curve(dev, cfg, row, grid, n_cb: int, seed: int):
    """Code-block error rate at each Es/N0 of `grid` (device encoder, channel and
    decoder; n_cb blocks of configuration cfg per point)."""
    import torch

    from deeplearning_5g_ldpc_decoder_b200 import channel_llrs, ldpc_decode, ldpc_encode

    gen = torch.Generator(device=dev).manual_seed(seed)
    pay = torch.randint(0, 256, (n_cb, cfg[1] // 8), dtype=torch.uint8, device=dev, generator=gen)
    rm = ldpc_encode(pay, cfg)
    out = []
    for k, snr in enumerate(grid):
        res = ldpc_decode(channel_llrs(rm, cfg[3], cfg[5], -float(snr), seed=seed * 1000 + k), cfg, row)
        ok = (res.status == 0) & (res.hardbits[:, : cfg[1] // 8] == pay).all(dim=1)
        out.append(1.0 - float(ok.float().mean()))
    return np.array(out)


def _calibrate_tb_snr10(dev, row, pool, n_cb: int = 2048):
    """Es/N0 of 10 % transport-block error for each MCS over the pool's own
    transport blocks.  Per MCS and base graph, the code-block error curve p(s)
    of one representative code block (BG1: A=8424, the size of every code
    block of a multi-block TB; BG2: A=1000) is measured on a 0.1 dB grid;
    transport block i with C_i code blocks fails with 1 - (1 - p(s))^C_i; the
    MCS's point is the Es/N0 where the mean over its blocks is 10 %."""
    rep = {1: 8424, 2: 1000}
    snr10 = {}
    for mi, (Qm, R) in enumerate(SERVE_MCS):
        members = [t for t in pool if t[0] == mi]
        if not members:
            continue
        shannon = 10 * np.log10(2 ** (Qm * R) - 1)
        grid = np.round(np.arange(shannon - 1.0, shannon + 7.0, 0.1), 2)
        curves = {}
        for bgn in sorted({t[1] for t in members}):
            A = rep[bgn]
            E = Qm * int(round((A + 24) / R / Qm))
            curves[bgn] = _cb_error_curve(dev, (bgn, A, 1, E, 0, Qm, 0), row, grid, n_cb, seed=17 + mi * 3 + bgn)
        vals = [float(np.mean([1.0 - (1.0 - curves[b][k]) ** C for _, b, C in members])) for k in range(len(grid))]
        # first grid point at or below 10 %, refined linearly from the point before it
        k = next((k for k, v in enumerate(vals) if v <= 0.1), len(grid) - 1)
        if k == 0:
            snr10[(Qm, R)] = float(grid[0])
        else:
            f = (vals[k - 1] - 0.1) / max(vals[k - 1] - vals[k], 1e-9)
            snr10[(Qm, R)] = float(grid[k - 1] + f * (grid[k] - grid[k - 1]))
    return snr10


def run_serve(args, loads=(10_000, 20_000, 50_000, 100_000, 200_000), pool_size: int = 1500,
              max_wait_s: float = 0.005):
    """Serving loop: Poisson transport-block arrivals at several offered loads
    through the native continuous-batching loop; p50/p99 verdict latency,
    achieved TB/s and decoded Gbit/s; the same blocks decoded through plain
    per-size launches for comparison."""
    import torch

    from deeplearning_5g_ldpc_decoder_b200 import ldpc_decode
    from deeplearning_5g_ldpc_decoder_b200 import tb as tbm

    row = [1, 10, 22936, 0, 1280, 32767, -32767]
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    rng = np.random.default_rng(2025)
    pool = args.n_cw if args.n_cw != N_CW else pool_size
    draws = []
    for _ in range(pool):
        A0 = float(np.exp(rng.uniform(np.log(200), np.log(1.2e6))))
        mi = int(rng.integers(len(SERVE_MCS)))
        Qm, R = SERVE_MCS[mi]
        bgn = tbm.select_bg(int(A0), R)
        A = tbm.round_tbs(A0, bgn)
        C, _ = tbm.code_block_count(A, bgn)
        G = tbm.coded_bits(A, bgn, Qm, R)
        if -(-G // Qm // C) * Qm > 65535:
            continue
        draws.append((mi, bgn, C, A, G, Qm))
    t_cal = time.perf_counter()
    snr10 = _calibrate_tb_snr10(dev, row, [(d[0], d[1], d[2]) for d in draws])
    t_cal = time.perf_counter() - t_cal
    rows, pays, noise, offset = [], [], [], []
    for mi, bgn, C, A, G, Qm in draws:
        rows.append((A, G, Qm, 0, bgn, 0, 0))
        pays.append(rng.integers(0, 256, A // 8, dtype=np.uint8))
        off = rng.uniform(-1.5, 1.5)   # 3 dB window around the MCS's 10 % transport-block error point
        offset.append(off)
        noise.append(-(snr10[SERVE_MCS[mi]] + off))
    offset = np.array(offset)
    t_enc = time.perf_counter()
    tbs, arena, out_bytes = tbm.encode_transport_blocks(pays, tbm.tb_array(rows), noise, seed=3, device=dev)
    torch.cuda.synchronize()
    t_enc = time.perf_counter() - t_enc
    n_pool = len(tbs)
    A_bits = tbs["A"].astype(np.int64)
    segs = [tbm.segment(int(t["A"]), int(t["G"]), int(t["Qm"]), int(t["bgn"]), int(t["rv"])) for t in tbs]
    n_cbs = np.array([s.C for s in segs])
    out = torch.zeros(out_bytes + 8, dtype=torch.uint8, device=dev)
    eng = tbm.TbEngine(max_tbs=8192, max_cbs=65536, decoder_row=row)
    stream = torch.cuda.Stream(dev)

    # offline: the whole pool in batches of the engine's size, and through plain per-size launches
    with torch.cuda.stream(stream):
        st_off, _ = eng.decode(tbs, arena, out)          # warm-up
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record(stream)
        for _ in range(max(1, args.steps // 4)):
            st_off, it_off = eng.decode(tbs, arena, out)
        e1.record(stream)
    stream.synchronize()
    ms_engine = e0.elapsed_time(e1) / max(1, args.steps // 4)
    st_off = st_off.cpu().numpy()
    groups = []
    for i, (t, s) in enumerate(zip(tbs, segs)):
        base = int(t["llr_offset"])
        for lo, hi in ((0, s.n_lo), (s.n_lo, s.C)):
            if hi > lo:
                E = s.E(lo)
                cfg = (s.cb_cfg[0], s.cb_cfg[1], s.cb_cfg[2], E, s.cb_cfg[4], s.cb_cfg[5], 0)
                start = base + s.llr_start(lo)
                groups.append((arena[start:start + (hi - lo) * E].view(hi - lo, E), cfg))
    with torch.cuda.stream(stream):
        for llr_g, cfg in groups[:64]:
            ldpc_decode(llr_g, cfg, row)
        e0.record(stream)
        for llr_g, cfg in groups:
            ldpc_decode(llr_g, cfg, row)
        e1.record(stream)
    stream.synchronize()
    ms_plain = e0.elapsed_time(e1)
    pool_gbit = float(A_bits.sum()) / 1e9

    results = []
    for lam in loads:
        n_arr = int(min(max(2000, lam * 0.25), 50_000))
        pick = rng.integers(0, n_pool, n_arr)
        trace = tbs[pick]
        arrivals = np.cumsum(rng.exponential(1.0 / lam, n_arr))
        with torch.cuda.stream(stream):
            res = tbm.serve(eng, trace, arrivals, arena, out, max_batch_tbs=8192, max_batch_cbs=65536,
                            llr_budget_bytes=4 << 30, pipeline_depth=args.pipeline_depth, timeout_s=120.0,
                            max_wait_s=max_wait_s, stream=stream)
        done = res.status >= 0
        lat = res.latency_s[done] * 1e3
        bits_ok = float(A_bits[pick][res.status == 0].sum())
        bits_done = float(A_bits[pick][done].sum())
        wall = res.stats["wall_s"]
        results.append({"offered_tb_per_s": lam, "tbs": n_arr, "admitted": int(res.stats["admitted"]),
                        "dropped": int(res.stats["dropped"]), "expired": int(res.stats["expired"]),
                        "achieved_tb_per_s": round(done.sum() / wall, 1),
                        "decoded_gbit_per_s": round(bits_done / wall / 1e9, 4),
                        "goodput_gbit_per_s": round(bits_ok / wall / 1e9, 4),
                        "latency_ms_p50": round(float(np.percentile(lat, 50)), 3),
                        "latency_ms_p99": round(float(np.percentile(lat, 99)), 3),
                        "tb_bler": round(float((res.status[done] != 0).mean()), 4),
                        "batches": int(res.stats["batches"]), "mean_batch_tbs": round(res.stats["mean_batch_tbs"], 1)})
    best = max(results, key=lambda d: d["decoded_gbit_per_s"])
    center = np.abs(offset) < 0.25
    return {"metric": "TB serving: decoded Gbit/s and p50/p99 TB latency", "value": best["decoded_gbit_per_s"],
            "unit": "Gbit/s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": round(ms_engine, 3), "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "int16",
            "data": "synthetic: device-encoded transport blocks, log-uniform 200..1.2M bits, 8 MCS over Qm {2,4,6,8}, "
                    "per-block Es/N0 uniform in +-1.5 dB around the MCS's 10 % transport-block error point "
                    "(calibrated on the device over the pool's own block sizes)",
            "config": {"workload": f"serving: pool of {n_pool} transport blocks ({int(n_cbs.sum())} code blocks, "
                                   f"{pool_gbit:.3f} Gbit), Poisson arrivals {loads[0] // 1000}k-{loads[-1] // 1000}k "
                                   f"TB/s, LLR budget 4 GiB, wait bound {max_wait_s * 1e3:g} ms, algo 1 10 iterations "
                                   f"with CRC early exit, continuous batching depth {args.pipeline_depth}",
                       "parallelism": "single GPU"},
            "loads": results,
            "offline_pool": {"engine_ms": round(ms_engine, 3), "engine_gbit_per_s": round(pool_gbit / ms_engine * 1e3, 4),
                             "plain_per_size_ms": round(ms_plain, 3),
                             "plain_per_size_gbit_per_s": round(pool_gbit / ms_plain * 1e3, 4),
                             "plain_launches": len(groups), "speedup": round(ms_plain / ms_engine, 2),
                             "tb_bler": round(float((st_off != 0).mean()), 4),
                             "tb_bler_window_center": round(float((st_off[center] != 0).mean()), 4),
                             "blocks_window_center": int(center.sum()),
                             "note": "a uniform +-1.5 dB window across a waterfall about 1 dB wide puts about half "
                                     "its blocks below the 10 % point, so the window's mean TB error is well above "
                                     "10 %; blocks within 0.25 dB of the centre sit near 10 %"},
            "mcs_tb_snr10_db": {f"Qm{q}_R{r}": round(v, 2) for (q, r), v in snr10.items()},
            "setup_s": {"calibration": round(t_cal, 1), "encode": round(t_enc, 1)},
            "gpu_launches": int(3 * sum(d["batches"] for d in results))}


TRAIN_CONFIGS = {"bg2_zc64": (2, 488, 1, 1920, 0, 2, 0), "bg1_zc112": (1, 2440, 1, 7392, 0, 2, 0)}


def _train_cpu_baseline(cfg, T: int, batch: int = 64) -> dict:
    """Forward + backward of the autograd restatement of the reference's unrolled
    min-sum model on the host cores (the computation the reference trains with),
    on a bounded batch."""
    import torch

    from oracle.minsum_torch import MinSumGraph, bce_loss, minsum_unrolled

    torch.set_num_threads(os.cpu_count() or 1)
    g = MinSumGraph(*cfg[:6])
    gen = torch.Generator().manual_seed(0)
    llr = (2.0 + 1.5 * torch.randn((batch, g.n), generator=gen))
    target = torch.zeros((batch, g.B))
    ra = torch.zeros((T, g.rows), requires_grad=True)
    rb = torch.full((T, g.rows), -3.0, requires_grad=True)

    def step():
        a = 0.5 + 0.5 * torch.sigmoid(ra)
        fin, _ = minsum_unrolled(g, llr, a, torch.sigmoid(rb))
        bce_loss(fin, target, g.B).backward()

    step()
    t0 = time.perf_counter()
    n = 0
    while n < 3 or time.perf_counter() - t0 < 10.0:
        step()
        n += 1
    dt = (time.perf_counter() - t0) / n
    return {"value": round(batch / dt, 2), "unit": "codewords/s", "cores": torch.get_num_threads(), "kind": "port",
            "sample": f"{n} forward+backward passes of batch {batch}, {T} iterations, torch autograd on host cores"}


def run_train(args):
    """Learned min-sum training step: device batch generation excluded, then
    forward kernel + BCE loss + backward kernel + Adam step, per batch of 4096."""
    import torch

    from deeplearning_5g_ldpc_decoder_b200 import capi
    from deeplearning_5g_ldpc_decoder_b200.train import (NeuralLayeredMinSumDecoder, decoder_loss,
                                                         ebn0_to_noise_power_db, make_training_batch)

    T = 10
    batch = args.n_cw if args.n_cw != N_CW else 4096
    dev = torch.device("cuda", 0)
    torch.cuda.set_device(dev)
    base = None
    if not args.no_parity:
        base = _train_cpu_baseline(TRAIN_CONFIGS["bg2_zc64"], T)
    legs = {}
    for name, cfg in TRAIN_CONFIGS.items():
        model = NeuralLayeredMinSumDecoder(cfg, num_iterations=T, alpha_mode="checkpoint", init_alpha=0.7,
                                           init_beta=0.02).to(dev)
        opt = torch.optim.Adam(model.parameters(), lr=1e-2)
        llr, target = make_training_batch(model, batch, ebn0_to_noise_power_db(1.5, cfg[5], model.B, cfg[3]), seed=3)
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
        fwd_ms = bwd_ms = 0.0

        def step(timed):
            nonlocal fwd_ms, bwd_ms
            opt.zero_grad(set_to_none=True)
            if timed:
                ev[0].record()
            _, final = model(llr, return_llr=True)
            loss = decoder_loss(final, target, model.B)
            if timed:
                ev[1].record()
            loss.backward()
            if timed:
                ev[2].record()
            opt.step()
            if timed:
                ev[3].record()
                torch.cuda.synchronize()
                fwd_ms += ev[0].elapsed_time(ev[1])
                bwd_ms += ev[1].elapsed_time(ev[2])

        for _ in range(max(args.warmup, 3)):
            step(False)
        torch.cuda.synchronize()
        l0 = capi.kernel_launch_count()
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        for _ in range(args.steps):
            step(False)
        t1.record()
        torch.cuda.synchronize()
        ms = t0.elapsed_time(t1) / args.steps
        launches = (capi.kernel_launch_count() - l0) // args.steps
        for _ in range(3):
            step(True)
        n = model.n
        ck_bytes = 4 * T * batch * sum(model.row_degrees) * model.Zc   # the tape of every edge's input
        legs[name] = {"ms_per_step": round(ms, 3), "codewords_per_s": round(batch / (ms * 1e-3), 1),
                      "forward_ms": round(fwd_ms / 3, 3), "backward_ms": round(bwd_ms / 3, 3),
                      "checkpoint_bytes": int(ck_bytes), "own_kernel_launches_per_step": int(launches),
                      "n": n, "Zc": model.Zc, "B": model.B}
    main = legs["bg2_zc64"]
    return {"metric": "learned min-sum training throughput", "value": main["codewords_per_s"],
            "unit": "codewords/s", "n_gpus": 1, "steps": args.steps, "warmup": args.warmup,
            "ms_per_step": main["ms_per_step"], "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "f32", "data": "synthetic: device-encoded random payloads, QPSK AWGN at Eb/N0 1.5 dB, int16 "
                                    "LLRs rate-recovered on device",
            "config": {"workload": f"learned min-sum training step, batch {batch}, {T} unrolled iterations, "
                                   "checkpoint alpha/beta; BG2 Zc64 (A=488, E=1920) headline, BG1 Zc112 beside",
                       "parallelism": "single GPU"},
            "legs": legs, "cpu_baseline": base, "gpu_launches": main["own_kernel_launches_per_step"] * args.steps}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--cpu-procs", type=int, default=0, help="host processes of the reference decode (0: all cores)")
    ap.add_argument("--no-parity", "--no-cpu-baseline", dest="no_parity", action="store_true",
                    help="skip the reference decode of the same blocks (parity and CPU baseline)")
    ap.add_argument("--n-cw", type=int, default=N_CW, help="code blocks per step (profiling runs use fewer)")
    ap.add_argument("--no-e2e", action="store_true", help="skip the host-buffer leg (profiling runs)")
    ap.add_argument("--no-legs", action="store_true", help="skip the mixed, serve and train legs of the default run")
    ap.add_argument("--algo", type=int, default=1, choices=[0, 1, 2, 3, 4],
                    help="decoder of the main step (profiling of the other kernels; the headline is algo 1)")
    ap.add_argument("--pipeline-depth", type=int, default=8, help="serve: batches in flight (streams)")
    ap.add_argument("--workload", default="bg1_zc384", choices=["bg1_zc384", "mixed", "train", "serve"],
                    help="mixed: 32768 blocks over all 51 lifting sizes, BG1 60 %%, rate U[0.2, 0.92], Qm 2-8; "
                         "train: learned min-sum forward+backward, batch 4096, 10 iterations")
    args = ap.parse_args()
    if args.gpus > 1 and "WORLD_SIZE" not in os.environ:
        # asked for N GPUs outside a launcher: start one rank per GPU here
        from deeplearning_5g_ldpc_decoder_b200.shard import launch_ranks

        sys.exit(launch_ranks(args.gpus, os.path.abspath(__file__), sys.argv[1:], timeout_s=1800))
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))

    if args.impl == "reference":
        if rank != 0:
            return
        llr = synthetic_llrs(args.n_cw, seed=0)
        ref = reference_decode(llr, CFG, ROW, procs=args.cpu_procs)
        base = cpu_baseline_from(ref, "the GPU arm's rank-0 step (seed 0, noisy, all 8 iterations run)")
        line = {
            "metric": METRIC, "value": round(base["value"], 6), "unit": "Gbit/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "int16", "impl": "reference",
            "data": (f"the GPU arm's own rank-0 LLRs: all {args.n_cw} blocks of synthetic_llrs(seed 0), random bits "
                     "on BPSK/AWGN at Eb/N0 0.9 dB (noisy, all 8 iterations run)"),
            "config": {"workload": WORKLOAD.replace("8192", str(args.n_cw)),
                       "parallelism": "one process per host core"},
            "cpu_baseline": base,
            "e2e": {"value": round(base["value"], 6), "unit": "Gbit/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0},
        }
        print(json.dumps(line), flush=True)
        return

    if args.workload == "mixed":
        if rank != 0:
            return
        print(json.dumps(run_mixed(args)), flush=True)
        return
    if args.workload == "train":
        if rank != 0:
            return
        print(json.dumps(run_train(args)), flush=True)
        return
    if args.workload == "serve":
        if rank != 0:
            return
        print(json.dumps(run_serve(args)), flush=True)
        return

    if world > 1:
        os.environ.setdefault("NCCL_DEBUG", "INFO")     # the communicator's rank count shows in the log
    result = run_gpu(args, rank, world, local_rank)
    if rank == 0:
        result.setdefault("cpu_baseline", None)
        if world == 1 and not args.no_e2e and not args.no_legs:
            # the other BASELINE workloads, each with its own clock record, as extra keys of the same line
            legs = (("mixed", lambda: run_mixed(args)),
                    ("serve", lambda: run_serve(args, loads=(10_000, 50_000, 200_000), pool_size=1000)),
                    ("train", lambda: run_train(args)))
            for name, fn in legs:
                sampler = ClockSampler()
                sampler.start()
                t0 = time.perf_counter()
                leg = fn()
                leg["clocks"] = sampler.stop()
                leg["leg_wall_s"] = round(time.perf_counter() - t0, 1)
                result[name] = leg
        print(json.dumps(result), flush=True)


if __name__ == "__main__":
    main()
