"""Benchmark of the imaginary-axis G0W0 hot path: G0W0 solves/s on one B200 per rank.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]
                    [--precision fp64|bf16x3] [--workload single840]

One step = one complete G0W0 solve (chi0 for all frequencies, eps(iw)
factorization, Sigma_c on the evaluation points, Pade continuation, graphical
QP equation) of the seeded synthetic instance Nocc=21, Nvirt=207, Naux=840,
32 imaginary frequencies, Sigma for HOMO and LUMO over all 228 states.
``value`` is the device-timed throughput with the inputs resident in HBM
(CUDA events around each solve on the library's stream, L2 flushed by a
512 MiB write between solves); ``e2e`` is the same solve through the host
pointer C-ABI call (pinned host inputs copied in, results copied out, inside the
timed region).  With N ranks (torchrun) every rank solves its own instance
(replicas, weak scaling); the time is the max over ranks.

``--impl reference`` times the CPU restatement of MOLGW's path (the oracle:
NumPy/SciPy on OpenBLAS, the reference's own BLAS/LAPACK call sequence) on the
host cores for the same instance and metric.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

HA_EV = 27.21138505
METRIC = "G0W0 solves/s"
WORKLOAD = "single synthetic RI-GW instance Nocc=21 Nvirt=207 Naux=840, 32 imaginary frequencies"
DATA = ("synthetic (seeded PCG64 seed 2 + rank; energies U[-30,-8]/U[0.5,40] eV, M ~ N(0,s^2) scaled so "
        "max eig eps(i0) = 1.8)")


def bench_config(precision: str, world: int) -> dict:
    """The ``config`` of the default line, printed identically by both arms."""
    return {"workload": WORKLOAD, "precision": precision,
            "parallelism": f"replicas x{world}" if world > 1 else "1 GPU",
            "l2": "flushed between solves (512 MiB write)", "sigma_states": "HOMO, LUMO",
            "nomega_sigma_calc": 50, "nomega_sigma": 101}


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=40)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--precision", default="fp64", choices=["fp64", "bf16x3"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--batch-count", type=int, default=256,
                    help="molecules of the ragged batch measured beside the single instance (0: skip)")
    ap.add_argument("--batch-reps", type=int, default=2, help="timed repetitions of the split-precision batch")
    ap.add_argument("--batch-reps-fp64", type=int, default=1, help="timed repetitions of the FP64 batch")
    ap.add_argument("--serving-window", type=float, default=10.0,
                    help="seconds of Poisson arrivals at --serve-rate in the default line's serving block (0: skip)")
    ap.add_argument("--serving-stable-rate", type=float, default=8.0,
                    help="arrival rate (req/s) of the sustainable-load run of the serving block")
    ap.add_argument("--serving-stable-window", type=float, default=20.0)
    ap.add_argument("--sweep-block", type=int, default=1,
                    help="1: add the precision-sweep instance (FP64, BF16x3, Ozaki 4) to the default line")
    ap.add_argument("--parallel", default="replicas", choices=["replicas", "frequencies"],
                    help="N > 1: independent replicas (weak scaling) or the frequencies of one molecule "
                         "sharded over the ranks with one all-reduce of Sigma_c (strong scaling)")
    ap.add_argument("--workload", default="single", choices=["single", "serve", "sweep", "aomo", "sox"])
    ap.add_argument("--sweep-reps", type=int, default=2)
    ap.add_argument("--serve-rate", type=float, default=200.0)
    ap.add_argument("--serve-duration", type=float, default=60.0)
    ap.add_argument("--serve-workers", type=int, default=2)
    ap.add_argument("--serve-batch", type=int, default=32)
    ap.add_argument("--serve-fp64", action="store_true", help="also serve the same arrivals in FP64")
    return ap.parse_args()


def chi0_flops(inst) -> float:
    """Algorithmic FLOPs of chi0 = M D M^T (symmetric rank-k update) over all frequencies."""
    nia = inst.nocc * inst.nvirt
    return float(inst.nomega) * inst.naux * (inst.naux + 1) * nia


def solve_flops(inst) -> float:
    n, p, s = inst.naux, inst.nstate, 2
    f_chi0 = chi0_flops(inst)
    f_eps = inst.nomega * (n ** 3 / 3.0 + n ** 3 / 3.0 + n * n * p * s)   # Cholesky + U^-T [I | M]
    return f_chi0 + f_eps


def oracle_solve(inst):
    from oracle import rigw_oracle as o
    rng = o.selfenergy_set_state_range(inst.nstate, inst.occupation, selfenergy_state_min=inst.nsemin,
                                       selfenergy_state_max=inst.nsemax)
    return o.g0w0_imag(inst.energy, inst.occupation, inst.m_ia, inst.m_sigma, inst.nomega, rng,
                       nomega_sigma=inst.nomega_sigma, step_sigma=inst.step_sigma,
                       nomega_sigma_calc=inst.nomega_sigma_calc, step_sigma_calc=inst.step_sigma_calc,
                       eta=inst.eta)


class ClockSampler:
    """SM clock, power and clock-event reasons sampled during the timed region.

    NVML is read from a thread every 10 ms (read-only queries), so a timed region
    of a tenth of a second still holds several samples; ``nvidia-smi -lms 200``
    is the fallback when NVML cannot be loaded.  The GPU is found by the PCI bus
    id of the CUDA device, so the samples are of the GPU that runs the work."""
    NAMES = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")

    def __init__(self, cuda_index: int, period_s: float = 0.01):
        self.cuda_index = cuda_index
        self.period = period_s
        self.samples = []            # (time, sm_mhz, max_mhz, power_w, reasons)
        self.thread = None
        self.smi = None

    def _handle(self):
        import pynvml
        pynvml.nvmlInit()
        try:
            import torch
            pr = torch.cuda.get_device_properties(self.cuda_index)
            bus = f"{pr.pci_domain_id:08x}:{pr.pci_bus_id:02x}:{pr.pci_device_id:02x}.0"
            return pynvml, pynvml.nvmlDeviceGetHandleByPciBusId(bus)
        except Exception:
            return pynvml, pynvml.nvmlDeviceGetHandleByIndex(self.cuda_index)

    def start(self):
        import threading
        try:
            nv, h = self._handle()
            bits = (nv.nvmlClocksEventReasonHwSlowdown, nv.nvmlClocksEventReasonHwThermalSlowdown,
                    nv.nvmlClocksEventReasonSwThermalSlowdown, nv.nvmlClocksEventReasonSwPowerCap)
            mx = float(nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM))
        except Exception:
            return self._start_smi()
        self.stop_flag = threading.Event()

        def loop():
            while not self.stop_flag.is_set():
                try:
                    sm = float(nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM))
                    pw = nv.nvmlDeviceGetPowerUsage(h) * 1e-3
                    rs = nv.nvmlDeviceGetCurrentClocksEventReasons(h)
                    self.samples.append((time.time(), sm, mx, pw,
                                         tuple(n for n, b in zip(self.NAMES, bits) if rs & b)))
                except Exception:
                    pass
                self.stop_flag.wait(self.period)
        self.thread = threading.Thread(target=loop, daemon=True)
        self.thread.start()

    def _start_smi(self):
        import tempfile
        q = ("timestamp,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
             "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
             "clocks_event_reasons.sw_power_cap")
        self.path = Path(os.environ.get("RIGW_CLOCKS_CSV", tempfile.gettempdir())) / f"clocks_{os.getpid()}.csv"
        try:
            self.f = open(self.path, "w")
            self.smi = subprocess.Popen(["nvidia-smi", f"--query-gpu={q}", "--format=csv,noheader,nounits",
                                         "-i", str(self.cuda_index), "-lms", "200"], stdout=self.f,
                                        stderr=subprocess.DEVNULL)
        except Exception:
            self.smi = None

    def mark(self, which: str):
        """Wall-clock bounds of the timed region (samples outside it are not used)."""
        setattr(self, which, time.time())

    def _collect_smi(self):
        import datetime
        self.smi.terminate()
        self.smi.wait(timeout=10)
        self.f.close()
        for r in self.path.read_text().strip().splitlines():
            c = [x.strip() for x in r.split(",")]
            if len(c) < 8:
                continue
            try:
                t = datetime.datetime.strptime(c[0], "%Y/%m/%d %H:%M:%S.%f").timestamp()
                self.samples.append((t, float(c[1]), float(c[2]), float(c[3]),
                                     tuple(n for n, v in zip(self.NAMES, c[4:8]) if v == "Active")))
            except ValueError:
                continue

    def stop(self) -> dict:
        if self.thread is not None:
            self.stop_flag.set()
            self.thread.join(timeout=5)
            src = "NVML every 10 ms"
        elif self.smi is not None:
            self._collect_smi()
            src = "nvidia-smi every 200 ms"
        else:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["clock sampling unavailable"]}
        t0, t1 = getattr(self, "begin", None), getattr(self, "end", None)
        rows = [r for r in self.samples if t0 is None or t1 is None or t0 <= r[0] <= t1]
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0, "source": src}
        return {"sm_mhz": statistics.median(r[1] for r in rows), "sm_max_mhz": max(r[2] for r in rows),
                "reasons": sorted({n for r in rows for n in r[4]}), "samples": len(rows),
                "power_w_max": max(r[3] for r in rows), "source": src,
                "window": "samples taken inside the timed region"}


FP64_DIGIT_PRODUCTS = 34   # int8 digit products of one FP64 product (seven digits, levels i + j <= 9)


def measured_fp64_peak(torch) -> float:
    """cuBLAS DGEMM throughput (TFLOP/s) on this GPU: 8192^3 float64, best of 5."""
    n = 8192
    a = torch.randn(n, n, dtype=torch.float64, device="cuda")
    b = torch.randn(n, n, dtype=torch.float64, device="cuda")
    best = 1e9
    for _ in range(6):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        torch.matmul(a, b)
        e1.record()
        torch.cuda.synchronize()
        best = min(best, e0.elapsed_time(e1))
    del a, b
    return 2.0 * n ** 3 / (best * 1e-3) / 1e12


def profile_traffic(name: str):
    """DRAM bytes per launch of a kernel from a committed ncu summary (profiles/*.txt)."""
    p = ROOT / "profiles" / name
    if not p.exists():
        return None
    for line in p.read_text().splitlines():
        if line.startswith("dram_bytes_per_launch_fullsize:"):
            try:
                return float(line.split(":")[1])
            except ValueError:
                return None
    return None


def compact_tuning(rep: dict) -> dict:
    """The autotuner's choice and its effect, without the candidate list."""
    return {k: rep[k] for k in ("chi0_rows", "update_rows", "split_group", "chains", "panel_group", "default_ms",
                                "tuned_ms")} | {
        "candidates": len(rep["candidates"])}


def run_batched(eng, count: int, reps: int, flush_l2, reps_fp64: int | None = None) -> dict:
    """The ragged batch (Nocc ~ U{5..60}, Nvirt = round(Nocc*U[8,10]), Naux =
    4(Nocc+Nvirt), 32 frequencies, seeds 4..) in one call, split precision and
    FP64, QP-only outputs; inputs generated and kept in device memory."""
    import torch
    from molgw_b200 import synth
    from molgw_b200.rigw import RIGW_BF16X3, RIGW_FP64
    sizes = synth.batch_sizes(count)
    insts, devs = [], []
    for (no, nv, na, nw, sd) in sizes:
        inst, dev = synth.make_instance_device(no, nv, na, nw, sd)
        insts.append(inst)
        devs.append(dev)
    torch.cuda.synchronize()
    res, outs = {}, {}
    tuning = {}
    for prec, name in ((RIGW_BF16X3, "bf16x3"), (RIGW_FP64, "fp64")):
        # the autotuner runs on the first 8 molecules; its choice applies to the whole batch
        tuning[name] = compact_tuning(eng.autotune(insts[:8], prec, devs[:8], qp_only=True))
        eng.g0w0_batch(insts, prec, devs, qp_only=True)
        dev_ms, wall_ms, stage_ms = [], [], []
        for _ in range(reps if (name == "bf16x3" or reps_fp64 is None) else reps_fp64):
            flush_l2()
            t0 = time.perf_counter()
            o = eng.g0w0_batch(insts, prec, devs, qp_only=True)
            wall_ms.append((time.perf_counter() - t0) * 1e3)
            st = eng.last_stats()
            dev_ms.append(st["total_ms"])
            stage_ms.append(st["stage_ms"])
        outs[name] = o
        res[name] = {"solves_per_s": count / (np.mean(dev_ms) * 1e-3),
                     "solves_per_s_wall": count / (np.mean(wall_ms) * 1e-3),
                     "ms_per_batch": float(np.mean(dev_ms)), "wall_ms_per_batch": float(np.mean(wall_ms)),
                     "stage_ms": dict(zip(("pack", "chi0", "eps_factor_solve", "sigma_qp"),
                                          np.mean(np.array(stage_ms), axis=0).round(3).tolist())),
                     "waves": st["waves"], "chunks": st["chunks"], "kernel_launches": st["kernel_launches"],
                     "tuning": tuning[name]}
    dqp = max(float(np.abs(a.energy_qp_g - b.energy_qp_g).max()) for a, b in zip(outs["fp64"], outs["bf16x3"]))
    res["qp_max_diff_mev_split_vs_fp64"] = dqp * HA_EV * 1e3
    res["speedup_split_vs_fp64"] = res["bf16x3"]["solves_per_s"] / res["fp64"]["solves_per_s"]
    res["workload"] = (f"{count} ragged molecules, seeds 4..{3 + count}: Nocc~U{{5..60}}, Nvirt=round(Nocc*U[8,10]), "
                       "Naux=4(Nocc+Nvirt), 32 frequencies, QP-only outputs, one call per batch")
    del devs
    torch.cuda.empty_cache()
    return res


def run_serving(rate: float, duration: float, precision: int, workers: int, max_batch: int,
                grace: float = 15.0) -> dict:
    """Poisson arrivals (rate req/s for `duration` s; 95% ragged sizes, 5% large
    Nocc=150/Nvirt=1500/Naux=6000/48 frequencies) submitted in real time to the
    request loop.  Latency = completion - scheduled arrival on the monotonic clock
    (the loop stamps completions itself).  The run ends when every request is
    done or `grace` s after the last arrival; requests still queued then are
    cancelled and enter the percentiles with their latency so far (a lower
    bound).  Request inputs come from a device-resident pool: one instance per
    Nocc class (Nvirt = 9 Nocc, Naux = 40 Nocc) and one large instance."""
    import torch
    from molgw_b200 import synth
    from molgw_b200.rigw import Server
    sched = synth.serving_sizes(rate=rate, duration=duration)
    pool = {}
    for _, (no, nv, na, nw, sd) in sched:
        key = (no, nw)
        if key not in pool:
            nv2 = nv if no == 150 else 9 * no
            pool[key] = synth.make_instance_device(no, nv2, 4 * (no + nv2), nw, 7000 + no)
    torch.cuda.synchronize()
    srv = Server(0, workers=workers, max_batch=max_batch)
    # warm the worker plans on one request of each kind
    warm = 0
    for key in list(pool)[:2]:
        srv.wait(srv.submit(pool[key][0], precision, pool[key][1], qp_only=True))
        warm += 1
    tickets, arrive, large = [], [], []
    t0 = time.monotonic_ns()
    for at, (no, nv, na, nw, sd) in sched:
        target = t0 + int(at * 1e9)
        now = time.monotonic_ns()
        if target > now:
            time.sleep((target - now) * 1e-9)
        inst, dev = pool[(no, nw)]
        tickets.append(srv.submit(inst, precision, dev, qp_only=True))
        arrive.append(target)
        large.append(no == 150)
    deadline = time.monotonic_ns() + int(grace * 1e9)
    while time.monotonic_ns() < deadline and srv.counters()["completed"] - warm < len(tickets):
        time.sleep(0.02)
    t_end = time.monotonic_ns()
    loop_stats = srv.stats()
    info = [srv.info(t) for t in tickets]
    lat = np.array([(d_ns if d else t_end) - a for (d, _, d_ns), a in zip(info, arrive)]) * 1e-6
    done = np.array([d for d, _, _ in info])
    outs = [srv.wait(t, 0.0) if d else None for t, d in zip(tickets, done)]
    last = max([d_ns for d, _, d_ns in info if d] or [t_end])
    srv.close()
    large = np.array(large)
    span = (max(last, arrive[-1]) - t0) * 1e-9

    def stats(mask):
        if not mask.any():
            return None
        return {"requests": int(mask.sum()), "completed": int((done & mask).sum()),
                "p50_ms": float(np.percentile(lat[mask], 50)), "p99_ms": float(np.percentile(lat[mask], 99))}
    return {"requests": len(tickets), "completed": int(done.sum()), "large_requests": int(large.sum()),
            "offered_rate": rate, "duration_s": duration, "grace_s": grace,
            "solves_per_s": float(done.sum()) / span, "p50_ms": float(np.percentile(lat, 50)),
            "p99_ms": float(np.percentile(lat, 99)), "max_ms": float(lat.max()), "span_s": span,
            "latency_note": "requests unfinished at the end enter with their latency so far (lower bound)",
            "small": stats(~large), "large": stats(large),
            "workers": workers, "max_batch": max_batch, "loop_stats": loop_stats, "outputs": outs, "pool": pool}


def run_serve_line(args):
    """`--workload serve`: the request loop under Poisson arrivals, split precision
    (and FP64 with --serve-fp64), one JSON line."""
    import torch
    from molgw_b200 import build
    build.build()
    from molgw_b200.rigw import RIGW_BF16X3, RIGW_FP64, Engine
    torch.cuda.set_device(0)
    res = {}
    split = run_serving(args.serve_rate, args.serve_duration, RIGW_BF16X3, args.serve_workers, args.serve_batch)
    pool, outs = split.pop("pool"), split.pop("outputs")
    res["bf16x3"] = split
    # accuracy: every distinct instance of the pool once in FP64 (single context)
    eng = Engine(0)
    sched = None
    worst = 0.0
    seen = {}
    from molgw_b200 import synth
    sched = synth.serving_sizes(rate=args.serve_rate, duration=args.serve_duration)
    for (at, (no, nv, na, nw, sd)), o in zip(sched, outs):
        if o is None:
            continue
        key = (no, nw)
        if key not in seen:
            inst, dev = pool[key]
            seen[key] = eng.g0w0(inst, RIGW_FP64, dev, qp_only=True)
        worst = max(worst, float(np.abs(o.energy_qp_g - seen[key].energy_qp_g).max() * HA_EV * 1e3))
    eng.close()
    res["bf16x3"]["qp_max_diff_mev_vs_fp64"] = worst
    if args.serve_fp64:
        del pool, outs
        torch.cuda.empty_cache()
        try:
            f64 = run_serving(args.serve_rate, args.serve_duration, RIGW_FP64, args.serve_workers, args.serve_batch)
            f64.pop("pool")
            f64.pop("outputs")
            res["fp64"] = f64
            res["speedup_split_vs_fp64"] = res["bf16x3"]["solves_per_s"] / f64["solves_per_s"]
        except Exception as exc:     # reported, not hidden
            res["fp64"] = {"error": str(exc)}
    line = {"metric": "G0W0 solves/s + p50/p99 latency (request loop)", "unit": "solves/s",
            "value": res["bf16x3"]["solves_per_s"], "n_gpus": 1, "higher_is_better": True, "dtype": "bf16x3+f64",
            "data": "synthetic (Poisson arrivals, seed 5; sizes snapped to Nocc classes)",
            "config": {"workload": "serving: Poisson arrivals, 95% ragged sizes / 5% Nocc=150 Nvirt=1500 Naux=6000 "
                                   "48 frequencies", "rate": args.serve_rate, "duration_s": args.serve_duration},
            "serving": res}
    print(json.dumps(line), flush=True)


def run_serving_block(args) -> dict:
    """The serving block of the default line (BASELINE config 5 in a shorter
    window): Poisson arrivals at ``--serve-rate`` req/s for ``--serving-window``
    s into the request loop, split precision and FP64 on the same arrivals, then
    a sustainable rate (``--serving-stable-rate``) in split precision.  p50/p99
    latency per lane and solves/s per precision; the QP difference in meV
    between the split and FP64 results of the requests both runs completed
    (same arrival schedule, same inputs)."""
    import torch
    from molgw_b200.rigw import RIGW_BF16X3, RIGW_FP64

    def run(rate, window, prec, grace):
        r = run_serving(rate, window, prec, args.serve_workers, args.serve_batch, grace=grace)
        r.pop("pool")
        outs = r.pop("outputs")
        r.pop("loop_stats", None)
        torch.cuda.empty_cache()
        return r, outs

    res = {"note": "latency = completion - scheduled arrival; requests unfinished at the end of the grace "
                   "period enter with their latency so far (lower bound)"}
    split, so = run(args.serve_rate, args.serving_window, RIGW_BF16X3, 5.0)
    f64, fo = run(args.serve_rate, args.serving_window, RIGW_FP64, 5.0)
    both = [(a, b) for a, b in zip(so, fo) if a is not None and b is not None]
    res["overload"] = {"rate": args.serve_rate, "window_s": args.serving_window, "bf16x3": split, "fp64": f64,
                       "speedup_split_vs_fp64": split["solves_per_s"] / f64["solves_per_s"],
                       "qp_max_diff_mev_split_vs_fp64": max(
                           (float(np.abs(a.energy_qp_g - b.energy_qp_g).max() * HA_EV * 1e3) for a, b in both),
                           default=None),
                       "compared_requests": len(both)}
    if args.serving_stable_rate > 0:
        stable, _ = run(args.serving_stable_rate, args.serving_stable_window, RIGW_BF16X3, 10.0)
        res["stable"] = {"rate": args.serving_stable_rate, "window_s": args.serving_stable_window,
                         "bf16x3": stable}
    return res


def h2o_instance():
    """The H2O cc-pVDZ G0W0@HF workload (HF in cc-pVDZ with cc-pVDZ-RI, 24
    functions, 84 auxiliary functions, 5 occupied, 16 frequencies, HOMO and
    LUMO) from its committed fixture, with the oracle's QP energies stored there."""
    from molgw_b200.synth import GWInstance
    d = np.load(ROOT / "tests" / "golden" / "h2o_ccpvdz.npz")
    c, b3 = d["c_matrix"], d["b3_ao"]
    m = np.einsum("ip,jq,ijP->pqP", c, c, b3, optimize=True)
    nocc = int(np.sum(d["occupation"] > 0))
    grid = {k: v for k, v in json.loads(str(d["workload_grid"])).items() if k != "nomega"}
    inst = GWInstance(nocc=nocc, nvirt=m.shape[0] - nocc, naux=m.shape[2], nomega=16, energy=d["energy"].copy(),
                      occupation=d["occupation"].copy(), m_ia=np.ascontiguousarray(m[:nocc, nocc:]),
                      m_sigma=np.ascontiguousarray(m[nocc - 1:nocc + 1]), nsemin=nocc, nsemax=nocc + 1, **grid)
    return inst, d["oracle_qp"]


def run_h2o_block(reps: int = 20, batch: int = 256) -> dict:
    """The H2O cc-pVDZ workload: one FP64 solve at a time through the host-pointer
    C ABI (wall time per call, host buffers, copies inside) and ``batch`` copies
    in one batched call; QP energies against the oracle's, stored in the fixture."""
    import torch
    from molgw_b200.rigw import Engine
    inst, ref_qp = h2o_instance()
    eng = Engine(0)
    for _ in range(3):
        out = eng.g0w0(inst)
    walls, dev = [], []
    for _ in range(reps):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        out = eng.g0w0(inst)
        walls.append((time.perf_counter() - t0) * 1e3)
        dev.append(eng.last_stats()["total_ms"])
    eng.g0w0_batch([inst] * batch)
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    outs = eng.g0w0_batch([inst] * batch)
    bwall = time.perf_counter() - t0
    eng.close()
    err = max(float(np.abs(o.energy_qp_g - ref_qp).max()) for o in [out] + outs) * HA_EV * 1e3
    return {"workload": "H2O HF cc-pVDZ (24 bf) / cc-pVDZ-RI (84), 5 occupied, 16 Gauss-Legendre frequencies, "
                        "HOMO+LUMO, FP64; inputs from the oracle's Gaussian front end (pinned on the reference's "
                        "H2O SCF and RI-MP2 known answers)",
            "single_wall_ms": float(np.median(walls)), "single_device_ms": float(np.median(dev)),
            "single_solves_per_s": 1e3 / float(np.median(walls)),
            "batch": batch, "batch_solves_per_s": batch / bwall,
            "homo_lumo_ev": [float(out.energy_qp_g[0] * HA_EV), float(out.energy_qp_g[1] * HA_EV)],
            "qp_error_mev_vs_oracle": err}


CONTOUR_GRID = dict(nomega_real=6, nomega_sigma=11, step_sigma=0.05, eta=0.001)


def contour_args(inst):
    """Contour-deformation arguments on a synthetic instance: its W window, its
    Sigma states (HOMO, LUMO) over every state p, its imaginary frequencies,
    and the real-axis settings of tests/inputs/h2o_gw_contour.in."""
    return (inst.energy, inst.occupation, inst.m_ia, inst.m_sigma, inst.nsemin, inst.nsemax, inst.nomega,
            CONTOUR_GRID["nomega_real"], CONTOUR_GRID["nomega_sigma"], CONTOUR_GRID["step_sigma"], CONTOUR_GRID["eta"])


def run_contour_block(reps: int = 3) -> dict:
    """G0W0 by contour deformation (rigw_gw_selfenergy_contour) on the 21/207/840
    instance: 32 imaginary and 6 real frequencies of W, low-rank W from the
    device eigensolver, Sigma_c on 11 real points per state, QP; wall time per
    call through the host-pointer ABI and the library's stage times."""
    import torch
    from molgw_b200 import synth
    from molgw_b200.rigw import Engine
    inst = synth.single_instance_840()
    eng = Engine(0)
    args = contour_args(inst)
    eng.g0w0_contour(*args)
    walls, stages = [], []
    for _ in range(reps):
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        out = eng.g0w0_contour(*args)
        walls.append((time.perf_counter() - t0) * 1e3)
        stages.append(eng.last_stats()["stage_ms"])
    eng.close()
    st = np.median(np.array(stages), axis=0)
    return {"workload": "contour deformation on Nocc=21 Nvirt=207 Naux=840 (seed 2): 32 imaginary + 6 real "
                        "frequencies, HOMO+LUMO on 11 real points (step 0.05 Ha), FP64",
            "wall_ms": float(np.median(walls)), "solves_per_s": 1e3 / float(np.median(walls)),
            "stage_ms": {"inputs": float(st[0]), "chi0": float(st[1]), "eigensolver": float(st[2]),
                         "sigma_qp": float(st[3])},
            "de_max_ha": float(out.de_max), "rank": [int(x) for x in out.rank],
            "homo_lumo_ev": [float(out.ehomo * HA_EV), float(out.elumo * HA_EV)], "_qp": out.energy_qp_g.tolist()}


def ri_cluster(nwater: int):
    """Shells of an nwater water cluster (3 Angstrom lattice) in cc-pVTZ with
    cc-pVTZ-RI, from the basis texts of the H2O fixture, and all its pairs."""
    from molgw_b200 import basis as B
    d = np.load(ROOT / "tests" / "golden" / "h2o_ccpvdz.npz")
    texts = json.loads(str(d["basis"]))
    atoms = B.water_cluster(nwater)
    sh = B.molecule_shells(atoms, {int(z): t for z, t in texts["cc-pVTZ"].items()})
    ax = B.molecule_shells(atoms, {int(z): t for z, t in texts["cc-pVTZ-RI"].items()})
    nbf = B.nfunctions(sh)
    pairs = np.array([(k, l) for l in range(1, nbf + 1) for k in range(1, l + 1)], dtype=np.int32)
    return sh, ax, pairs


def run_ri_block(reps: int = 2) -> dict:
    """RI integrals on the device (rigw_eri_3center_raw and rigw_eri_3center) for
    water clusters in cc-pVTZ / cc-pVTZ-RI: wall time per call with the result in
    host memory, and of the raw call writing into device memory (median of
    ``reps`` after one untimed call)."""
    import torch
    from molgw_b200.rigw import Engine
    eng = Engine(0)
    out = {"workload": "(H2O)_n on a 3 Angstrom lattice, cc-pVTZ with cc-pVTZ-RI, all basis-function pairs, FP64",
           "clusters": []}
    for nw in (2, 8):
        sh, ax, pairs = ri_cluster(nw)
        naux = int(sum(2 * x.am + 1 for x in ax))
        dev = torch.empty((naux, len(pairs)), dtype=torch.float64, device="cuda")
        eng.eri_3center_raw(sh, ax, pairs)
        raw_t, dev_t, full_t = [], [], []
        for _ in range(reps):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            eng.eri_3center_raw(sh, ax, pairs)
            raw_t.append(time.perf_counter() - t0)
            t0 = time.perf_counter()
            eng.eri_3center_raw(sh, ax, pairs, out=dev)
            dev_t.append(time.perf_counter() - t0)
            t0 = time.perf_counter()
            e3 = eng.eri_3center(sh, ax, pairs)
            full_t.append(time.perf_counter() - t0)
        out["clusters"].append({"waters": nw, "nbf": int(sum(2 * x.am + 1 for x in sh)), "naux": naux,
                                "npair": int(len(pairs)), "nauxil_kept": int(e3.shape[0]),
                                "raw_3center_s": float(np.median(raw_t)),
                                "raw_3center_device_result_s": float(np.median(dev_t)),
                                "eri_3center_with_metric_s": float(np.median(full_t))})
        del dev
    eng.close()
    return out


def run_ao_to_qp_block(reps: int = 3) -> dict:
    """From the AO tensor to the QP energies for the 21/207/840/32 workload:
    B(mu nu, P) over all 26 106 pairs of nbf = 228 functions (N(0, s^2), s the
    scale of the 840 instance's M, so that M = C B C^T has its statistics), C
    orthonormal, the instance's energies; wall time per solve from a page-locked
    host AO tensor.  "device": Engine.g0w0_from_ao (one upload of the AO tensor,
    both transforms and the solve on the device).  "host": the two host-pointer
    transforms (each uploads the AO tensor) and the host-pointer solve (uploads M)."""
    import torch
    from molgw_b200 import synth
    from molgw_b200.rigw import Engine
    inst = synth.single_instance_840()
    nbf, naux, nocc = inst.nstate, inst.naux, inst.nocc
    rng = np.random.default_rng(228)
    pairs = np.array([(k, l) for l in range(1, nbf + 1) for k in range(1, l + 1)], dtype=np.int32)
    eri3 = pinned_copy(rng.standard_normal((naux, len(pairs))) * float(inst.m_ia.std()))
    c = np.linalg.qr(rng.standard_normal((nbf, nbf)))[0].T.copy()
    grid = dict(nomega_sigma=inst.nomega_sigma, step_sigma=inst.step_sigma, nomega_sigma_calc=inst.nomega_sigma_calc,
                step_sigma_calc=inst.step_sigma_calc, eta=inst.eta)
    eng = Engine(0)

    def device_path():
        return eng.g0w0_from_ao(eri3, pairs, c, inst.energy, inst.occupation, inst.nomega, inst.nsemin,
                                inst.nsemax, **grid)

    def host_path():
        from dataclasses import replace
        m_ia = eng.calculate_eri_3center_mo(eri3, pairs, c, nocc + 1, nbf, 1, nocc)
        m_pm = eng.calculate_eri_3center_mo(eri3, pairs, c, 1, nbf, inst.nsemin, inst.nsemax)
        return eng.g0w0(replace(inst, m_ia=m_ia, m_sigma=m_pm))

    res = {}
    outs = {}
    for name, fn in (("device", device_path), ("host", host_path)):
        fn()
        walls = []
        for _ in range(reps):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            outs[name] = fn()
            walls.append((time.perf_counter() - t0) * 1e3)
        res[name] = {"wall_ms": float(np.median(walls)), "solves_per_s": 1e3 / float(np.median(walls))}
    eng.close()
    small = 8 * (2 * nbf + nbf * nbf * 2)
    res["device"]["h2d_bytes"] = int(eri3.nbytes) + small
    res["host"]["h2d_bytes"] = 2 * int(eri3.nbytes) + small + 8 * naux * (nocc * (nbf - nocc) + 2 * nbf)
    res["qp_diff_mev_device_vs_host"] = float(np.abs(outs["device"].energy_qp_g - outs["host"].energy_qp_g).max()
                                              * HA_EV * 1e3)
    res["workload"] = (f"AO tensor of nbf={nbf}, Naux={naux} ({len(pairs)} pairs, {eri3.nbytes / 1e6:.0f} MB, "
                       "page-locked) to QP energies, Nocc=21, 32 frequencies, FP64")
    return res


def run_sweep_block(fp64_peak: float, bf16_peak: float) -> dict:
    """The precision-sweep instance of the default line (Nocc=100, Nvirt=1100,
    Naux=4000, 48 frequencies, seed 3, in device memory): one timed solve each in
    FP64, BF16x3 and Ozaki INT8 with 4 slices after one untimed solve, QP-only
    outputs, QP energies in meV and E_RPA against the FP64 solve of the same run."""
    import torch
    from molgw_b200 import synth
    from molgw_b200.rigw import RIGW_BF16X3, RIGW_FP64, RIGW_OZAKI, Engine
    no, nv, na, nw = 100, 1100, 4000, 48
    inst, dev = synth.make_instance_device(no, nv, na, nw, 3)
    torch.cuda.synchronize()
    f_chi0 = float(nw) * na * (na + 1) * (no * nv)
    out, ref = {}, None
    for name, prec, products, peak in (("fp64", RIGW_FP64, FP64_DIGIT_PRODUCTS, 2.0 * bf16_peak),
                                       ("bf16x3", RIGW_BF16X3, 3, bf16_peak),
                                       ("ozaki4", RIGW_OZAKI(4), 10, 2.0 * bf16_peak)):
        eng = Engine(0)
        eng.g0w0(inst, prec, dev, qp_only=True)
        o = eng.g0w0(inst, prec, dev, qp_only=True)
        st = eng.last_stats()
        eng.close()
        if ref is None:
            ref = o
        ach = f_chi0 / (st["stage_ms"][1] * 1e-3) / 1e12
        out[name] = {"ms_per_solve": st["total_ms"], "solves_per_s": 1e3 / st["total_ms"],
                     "stage_ms": st["stage_ms"], "chi0_tflops_algorithmic": ach,
                     "chi0_frac_of_peak": ach * products / peak, "tensor_products": products,
                     "qp_diff_mev_vs_fp64": float(np.abs(o.energy_qp_g - ref.energy_qp_g).max() * HA_EV * 1e3),
                     "erpa_rel_diff_vs_fp64": float(abs(o.erpa - ref.erpa) / abs(ref.erpa))}
    del dev
    torch.cuda.empty_cache()
    out["speedup_bf16x3_vs_fp64"] = out["fp64"]["ms_per_solve"] / out["bf16x3"]["ms_per_solve"]
    out["workload"] = "Nocc=100 Nvirt=1100 Naux=4000, 48 imaginary frequencies, QP-only (precision sweep instance)"
    return out


def run_sweep_line(args):
    """`--workload sweep`: the precision sweep on one large instance (Nocc=100,
    Nvirt=1100, Naux=4000, 48 frequencies, seed 3, generated in device memory):
    FP64, BF16x3 and Ozaki INT8 with 3..7 slices.  chi0 runs in the named
    arithmetic, the eps factorization, Sigma and the QP solve in FP64; QP energies
    are reported in meV against the FP64 solve of the same run.  One JSON line."""
    import torch
    from molgw_b200 import build, synth
    build.build()
    from molgw_b200.rigw import RIGW_BF16X3, RIGW_FP64, RIGW_OZAKI, Engine
    peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
    bf16_peak = float(peaks.get("bf16_tflops", 1590.0))
    fp64_peak = measured_fp64_peak(torch)
    no, nv, na, nw = 100, 1100, 4000, 48
    inst, dev = synth.make_instance_device(no, nv, na, nw, 3)
    torch.cuda.synchronize()
    f_chi0 = float(nw) * na * (na + 1) * (no * nv)
    clocks = ClockSampler(0)
    clocks.start()
    out, ref = {}, None
    plan = [("fp64", RIGW_FP64, FP64_DIGIT_PRODUCTS, 2.0 * bf16_peak,
             "2 x MEASURED_PEAKS.json bf16_tflops (34 int8 digit products)"),
            ("bf16x3", RIGW_BF16X3, 3, bf16_peak, "MEASURED_PEAKS.json bf16_tflops")]
    plan += [(f"ozaki{k}", RIGW_OZAKI(k), FP64_DIGIT_PRODUCTS if k == 7 else k * (k + 1) // 2, 2.0 * bf16_peak,
              "2 x MEASURED_PEAKS.json bf16_tflops (dense int8 rate = 2 x bf16 on B200)") for k in range(3, 8)]
    for name, prec, products, peak, peak_src in plan:
        eng = Engine(0)                 # one context per precision: its plan is freed before the next
        eng.g0w0(inst, prec, dev, qp_only=True)
        tot, chi = [], []
        for _ in range(args.sweep_reps):
            o = eng.g0w0(inst, prec, dev, qp_only=True)
            st = eng.last_stats()
            tot.append(st["total_ms"])
            chi.append(st["stage_ms"][1])
        eng.close()
        if ref is None:
            ref = o
        chi_ms = float(np.mean(chi))
        achieved = f_chi0 / (chi_ms * 1e-3) / 1e12
        out[name] = {"solves_per_s": 1e3 / float(np.mean(tot)), "ms_per_solve": float(np.mean(tot)),
                     "chi0_ms": chi_ms, "stage_ms": st["stage_ms"],
                     "chi0_tflops_algorithmic": achieved,
                     "chi0_tensor_ops_per_s": achieved * products, "tensor_products": products,
                     "chi0_frac_of_peak": achieved * products / peak, "peak": peak, "peak_source": peak_src,
                     "qp_diff_mev_vs_fp64": float(np.abs(o.energy_qp_g - ref.energy_qp_g).max() * HA_EV * 1e3),
                     "erpa_rel_diff_vs_fp64": float(abs(o.erpa - ref.erpa) / abs(ref.erpa))}
    clk = clocks.stop()
    line = {"metric": METRIC, "value": out["fp64"]["solves_per_s"], "unit": "solves/s", "n_gpus": 1,
            "steps": args.sweep_reps, "warmup": 1, "ms_per_step": out["fp64"]["ms_per_solve"],
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded torch.Generator in device memory; energies U[-30,-8]/U[0.5,40] eV, "
                    "M ~ N(0,s^2) scaled so max eig eps(i0) = 1.8)",
            "config": {"workload": "precision sweep: Nocc=100 Nvirt=1100 Naux=4000, 48 imaginary frequencies, "
                                   "QP-only outputs (HOMO/LUMO); value = the FP64 solve",
                       "chi0_flops_algorithmic": f_chi0, "l2": "inputs larger than L2 (M is 3.5 GB)"},
            "precisions": out, "clocks": clk}
    print(json.dumps(line), flush=True)


def run_aomo_line(args):
    """`--workload aomo`: the RI AO->MO transform (calculate_eri_3center_mo) through
    the host-pointer C ABI, FP64, BF16x3 and Ozaki INT8 (4 slices), for the two
    calls of a G0W0 run: the W window (m = virtual, n = occupied) and the Sigma
    states (m = all, n = HOMO, LUMO).  Sizes: nbf = Nocc + Nvirt with the 840
    instance's Nocc=21/Nvirt=207/Naux=840, and nbf=600/Naux=2000 with 50
    occupied states; B(mu nu, P) ~ N(0,1) over all pairs, C orthonormal.  The
    device times come from the library's CUDA events: upload + unpack of the AO
    tensor, the two products (with the operand splits), download.  TFLOP/s use
    F = Naux (4 npair n + 2 n m nbf), the algorithmic count of the two products.
    One JSON line."""
    import torch
    from molgw_b200 import build
    build.build()
    from molgw_b200.rigw import RIGW_BF16X3, RIGW_FP64, RIGW_OZAKI, Engine
    peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
    bf16_peak = float(peaks.get("bf16_tflops", 1590.0))
    fp64_peak = measured_fp64_peak(torch)
    eng = Engine(0)
    cases = []
    for (nbf, naux, nocc) in ((228, 840, 21), (600, 2000, 50)):
        rng = np.random.default_rng(nbf)
        pairs = np.array([(k, l) for l in range(1, nbf + 1) for k in range(1, l + 1)], dtype=np.int32)
        eri3 = rng.standard_normal((naux, len(pairs)))
        c = np.linalg.qr(rng.standard_normal((nbf, nbf)))[0].T.copy()
        for call, (m0, m1, n0, n1) in (("W window", (nocc + 1, nbf, 1, nocc)),
                                       ("Sigma states", (1, nbf, nocc, nocc + 1))):
            mc, nc = m1 - m0 + 1, n1 - n0 + 1
            flops = float(naux) * (4.0 * len(pairs) * nc + 2.0 * nc * mc * nbf)
            res, ref = {}, None
            for name, prec, products, peak in (("fp64", RIGW_FP64, 1, fp64_peak),
                                               ("bf16x3", RIGW_BF16X3, 3, bf16_peak),
                                               ("ozaki4", RIGW_OZAKI(4), 10, 2.0 * bf16_peak)):
                eng.calculate_eri_3center_mo(eri3, pairs, c, m0, m1, n0, n1, precision=prec)
                walls, stats = [], []
                for _ in range(3):
                    t0 = time.perf_counter()
                    o = eng.calculate_eri_3center_mo(eri3, pairs, c, m0, m1, n0, n1, precision=prec)
                    walls.append((time.perf_counter() - t0) * 1e3)
                    stats.append(eng.last_stats())
                if ref is None:
                    ref = o
                best = int(np.argmin([st["stage_ms"][1] for st in stats]))
                st = stats[best]
                prod_ms = st["stage_ms"][1]
                tf = flops / (prod_ms * 1e-3) / 1e12
                res[name] = {"wall_ms": float(min(walls)), "device_ms": st["total_ms"],
                             "upload_unpack_ms": st["stage_ms"][0], "products_ms": prod_ms,
                             "download_ms": st["stage_ms"][2], "products_tflops_algorithmic": tf,
                             "frac_of_peak": tf * products / peak, "tensor_products": products,
                             "rel_err_vs_fp64": float(np.abs(o - ref).max() / np.abs(ref).max())}
            cases.append({"nbf": nbf, "naux": naux, "npair": len(pairs), "call": call, "m": [m0, m1], "n": [n0, n1],
                          "flops_algorithmic": flops, "precisions": res})
    eng.close()
    w = cases[0]["precisions"]["fp64"]
    line = {"metric": "AO->MO transforms/s", "value": 1e3 / w["wall_ms"], "unit": "transforms/s", "n_gpus": 1,
            "steps": 3, "warmup": 1, "ms_per_step": w["wall_ms"], "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64",
            "data": "synthetic (seeded PCG64; B ~ N(0,1) over all basis pairs, C orthonormal)",
            "config": {"workload": "RI AO->MO transform through the host-pointer C ABI (host arrays in and out); "
                                   "value = the W-window call of the nbf=228/Naux=840 case in FP64",
                       "fp64_peak_tflops": fp64_peak, "bf16_peak_tflops": bf16_peak},
            "cases": cases}
    print(json.dumps(line), flush=True)


def pinned_copy(a: np.ndarray) -> np.ndarray:
    """A float64 copy of ``a`` in page-locked host memory (a view of a pinned
    torch tensor), so that host-pointer calls upload it at full PCIe speed."""
    import torch
    t = torch.empty(a.shape, dtype=torch.float64, pin_memory=True)
    out = t.numpy()
    out[...] = a
    return out


def run_sox_line(args):
    """`--workload sox`: GW+SOX on the imaginary axis (postscf 'GW+SOX_PADE').
    Sigma^SOX (sox_selfenergy_imag_grid) through the host-pointer C ABI on the
    Nocc=21/Nvirt=207/Naux=840 instance and on Nocc=50/Nvirt=500/Naux=2000 (50
    evaluation points each): the (p q|j c) product on the DMMA tile engine,
    F = 2 nsig (Nocc+Nvirt) Nocc Nvirt Naux, and the frequency sums in
    (element x point)/s over Nocc^2 Nvirt + Nocc Nvirt (Nvirt+1)/2 elements per
    state; the oracle's Sigma^SOX timed on the host cores beside it.  value = the
    whole GW+SOX solve (W, Sigma_c, Sigma^SOX, Pade, QP) per second on the 840
    instance through the host-pointer calls.  "sosex": Sigma^SOSEX from the
    resident W on the 840 instance with its full window tensor
    (synth.with_window), timed and checked against the oracle.  One JSON line."""
    import torch
    from threadpoolctl import threadpool_limits
    from molgw_b200 import build, synth
    build.build()
    from molgw_b200.rigw import Engine, efermi_of
    from oracle import rigw_oracle as o
    from dataclasses import replace
    fp64_peak = measured_fp64_peak(torch)
    eng = Engine(0)

    def pinned(inst):
        # the caller's M tensors in page-locked host memory, as in the default line's e2e
        return replace(inst, m_ia=pinned_copy(inst.m_ia), m_sigma=pinned_copy(inst.m_sigma))

    cases = []
    for name, inst in (("840", synth.single_instance_840()), ("2000", synth.make_instance(50, 500, 2000, 32, seed=1))):
        inst = pinned(inst)
        z = efermi_of(inst) + 1j * inst.step_sigma_calc * np.arange(inst.nomega_sigma_calc)
        for _ in range(2):
            out = eng.sox_selfenergy_imag_grid(inst, z)
        walls, stats = [], []
        for _ in range(max(3, args.steps)):
            t0 = time.perf_counter()
            out = eng.sox_selfenergy_imag_grid(inst, z)
            walls.append((time.perf_counter() - t0) * 1e3)
            stats.append(eng.last_stats())
        st = min(stats, key=lambda s: s["total_ms"])
        no, nv = inst.m_ia.shape[0], inst.m_ia.shape[1]
        nsig, ng = inst.m_sigma.shape[0], inst.m_sigma.shape[1]
        flops = 2.0 * nsig * ng * no * nv * inst.naux
        elems = nsig * (no * no * nv + no * nv * (nv + 1) / 2)
        window = inst.energy[:ng]
        with threadpool_limits(limits=os.cpu_count() or 1):
            t0 = time.perf_counter()
            ref = o.sox_selfenergy_imag(window, inst.m_sigma, inst.m_ia, z)
            cpu_ms = (time.perf_counter() - t0) * 1e3
        tf = flops / (st["stage_ms"][1] * 1e-3) / 1e12
        cases.append({"instance": name, "nocc": no, "nvirt": nv, "naux": inst.naux, "nsig": nsig, "points": int(z.size),
                      "wall_ms": float(min(walls)), "device_ms": st["total_ms"],
                      "upload_transpose_ms": st["stage_ms"][0], "product_ms": st["stage_ms"][1],
                      "product_tflops": tf, "product_frac_of_measured_fp64": tf / fp64_peak,
                      "sums_ms": st["stage_ms"][3],
                      "sums_gelem_points_per_s": elems * z.size / (st["stage_ms"][3] * 1e-3) / 1e9,
                      "max_abs_diff_vs_oracle_rel": float(np.abs(out - ref).max() / np.abs(ref).max()),
                      "oracle_ms": cpu_ms})
    inst = pinned(synth.single_instance_840())
    eng.gw_sox_imag(inst)
    walls = []
    for _ in range(max(3, args.steps)):
        t0 = time.perf_counter()
        res = eng.gw_sox_imag(inst)
        walls.append((time.perf_counter() - t0) * 1e3)
    gw = eng.g0w0(inst)
    shift = float(np.abs(res.energy_qp_g - gw.energy_qp_g).max() * HA_EV)
    # Sigma^SOSEX from the resident W on the same instance with a full window tensor
    inst_w, m_full = synth.with_window(synth.single_instance_840(), seed=3)
    m_full = pinned_copy(m_full)
    z = efermi_of(inst_w) + 1j * inst_w.step_sigma_calc * np.arange(inst_w.nomega_sigma_calc)
    _, _, wpol = eng.polarizability_grid_scalapack(inst_w)
    try:
        eng.sosex_selfenergy_imag_grid(wpol, inst_w, m_full, z)
        stats, walls_x = [], []
        for _ in range(3):
            t0 = time.perf_counter()
            out = eng.sosex_selfenergy_imag_grid(wpol, inst_w, m_full, z)
            walls_x.append((time.perf_counter() - t0) * 1e3)
            stats.append(eng.last_stats())
    finally:
        wpol.release()
    st = min(stats, key=lambda s: s["total_ms"])
    no, e = inst_w.nocc, inst_w.energy
    om, wt = o.imaginary_quad_grid(inst_w.nomega)
    with threadpool_limits(limits=os.cpu_count() or 1):
        t0 = time.perf_counter()
        sf = o.polarizability_grid(inst_w.m_ia, e[:no], e[no:], inst_w.occupation[:no], inst_w.occupation[no:], om, wt)
        ref = o.sosex_selfenergy_imag(e, m_full, no, list(range(inst_w.nsemin - 1, inst_w.nsemax)), sf.chi, sf.omega,
                                      sf.weight_quad, z)
        cpu_ms = (time.perf_counter() - t0) * 1e3
    sosex = {"instance": "840 (window tensor 350 MB, page-locked)", "wall_ms": float(min(walls_x)),
             "device_ms": st["total_ms"], "upload_transpose_ms": st["stage_ms"][0],
             "products_and_k_ms": st["stage_ms"][1], "sums_ms": st["stage_ms"][3],
             "max_abs_diff_vs_oracle_rel": float(np.abs(out - ref).max() / np.abs(ref).max()),
             "oracle_ms_incl_w": cpu_ms}
    eng.close()
    ms = float(np.median(walls))
    line = {"metric": "GW+SOX solves/s", "value": 1e3 / ms, "unit": "solves/s", "n_gpus": 1,
            "steps": max(3, args.steps), "warmup": 1, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f64", "data": "synthetic (seeded instances of molgw_b200.synth)",
            "config": {"workload": "GW+SOX on the imaginary axis through the host-pointer calls (M tensors in "
                                   "page-locked host memory), Nocc=21 Nvirt=207 Naux=840, 32 imaginary frequencies, "
                                   "50 evaluation points",
                       "fp64_peak_tflops": fp64_peak},
            "sox_qp_shift_ev": shift, "cases": cases, "sosex": sosex}
    print(json.dumps(line), flush=True)


def run_frequency_sharded(args, rank, world, local):
    """`--parallel frequencies`: each step is one G0W0 solve of the 21/207/840/32
    instance with its 32 frequencies sharded over the ranks (round robin, MOLGW's
    poorman split): W and Sigma_c of the rank's frequencies on its GPU, one NCCL
    all-reduce of the partial Sigma_c and energies, the QP equation on the sum
    (parallel.g0w0_frequency_sharded; the library calls are synchronous, so
    CUDA events recorded after a device synchronisation bracket the whole step).
    Strong scaling: the total work per step is fixed."""
    import torch
    import torch.distributed as dist
    from molgw_b200 import parallel, synth
    from molgw_b200.rigw import RIGW_FP64, Engine
    inst = synth.single_instance_840()
    eng = Engine(local)
    ref = eng.g0w0(inst) if rank == 0 else None
    for _ in range(args.warmup):
        parallel.g0w0_frequency_sharded(eng, inst, RIGW_FP64)
    dist.barrier()
    torch.cuda.synchronize()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(args.steps):
        out = parallel.g0w0_frequency_sharded(eng, inst, RIGW_FP64)
    torch.cuda.synchronize()
    e1.record()
    torch.cuda.synchronize()
    t = torch.tensor([e0.elapsed_time(e1)], device="cuda", dtype=torch.float64)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    total_ms = float(t.item())
    eng.close()
    if rank == 0:
        line = {"metric": METRIC, "value": args.steps / (total_ms * 1e-3), "unit": "solves/s", "n_gpus": world,
                "steps": args.steps, "warmup": args.warmup, "ms_per_step": total_ms / args.steps,
                "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": "f64", "data": DATA,
                "config": {**bench_config("fp64", world), "parallelism": f"frequencies over {world} ranks"},
                "qp_diff_mev_vs_one_gpu": float(np.abs(out.energy_qp_g - ref.energy_qp_g).max() * HA_EV * 1e3),
                "timing": "CUDA events around the steps after device synchronisation (synchronous library calls), "
                          "max over ranks"}
        if isinstance(line.get("contour"), dict):
            line["contour"].pop("_qp", None)
        print(json.dumps(line), flush=True)
    dist.barrier()
    dist.destroy_process_group()


def run_reference(args, rank, world):
    """CPU restatement of the MOLGW path on the host cores (rank 0 only)."""
    if rank != 0:
        return
    from threadpoolctl import threadpool_limits
    from molgw_b200 import synth
    cores = os.cpu_count() or 1
    inst = synth.single_instance_840()
    times = []
    with threadpool_limits(limits=cores):
        for i in range(args.warmup + args.steps):
            t0 = time.perf_counter()
            oracle_solve(inst)
            dt = time.perf_counter() - t0
            if i >= args.warmup:
                times.append(dt)
    mean = sum(times) / len(times)
    value = 1.0 / mean
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": mean * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": DATA,
        "config": bench_config("fp64", args.gpus),
        "latency_ms": {"p50": float(np.percentile(times, 50) * 1e3), "p99": float(np.percentile(times, 99) * 1e3)},
        "cpu_baseline": {"value": value, "unit": "solves/s", "cores": cores, "kind": "port",
                         "sample": "full G0W0 solves of the same instance (CPU restatement of MOLGW's "
                                   "DSYRK/DSYEV/DGETRF/DGETRI/DGEMM path, OpenBLAS threads)"},
        "e2e": {"value": value, "unit": "solves/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def main():
    args = parse()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank, world)
        return
    if args.workload == "sweep":
        if args.impl == "reference":
            print(json.dumps({"impl": "reference", "unavailable": "the CPU restatement of one Naux=4000 solve "
                              "(84 TFLOP of chi0) does not finish in minutes"}), flush=True)
            return
        run_sweep_line(args)
        return
    if args.workload == "serve":
        run_serve_line(args)
        return
    if args.workload == "aomo":
        run_aomo_line(args)
        return
    if args.workload == "sox":
        run_sox_line(args)
        return

    import torch
    import torch.distributed as dist
    from datetime import timedelta

    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", timeout=timedelta(seconds=120))

    from molgw_b200 import build, synth
    if rank == 0 or world == 1:
        build.build()
    if world > 1:
        dist.barrier()
    from molgw_b200.rigw import RIGW_BF16X3, RIGW_FP64, Engine

    if args.parallel == "frequencies" and world > 1:
        run_frequency_sharded(args, rank, world, local)
        return
    precision = RIGW_FP64 if args.precision == "fp64" else RIGW_BF16X3
    inst = synth.single_instance_840(seed=2 + rank)
    eng = Engine(local)

    # inputs resident in HBM
    nocc = inst.nocc
    e, occ = inst.energy, inst.occupation
    host_arrays = {"m_ia": inst.m_ia, "e_occ": e[:nocc], "e_virt": e[nocc:], "occ_occ": occ[:nocc],
                   "occ_virt": occ[nocc:], "m_pm": inst.m_sigma, "e_p": e,
                   "e_sig": e[inst.nsemin - 1:inst.nsemax], "occ_sig": occ[inst.nsemin - 1:inst.nsemax]}
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda() for k, v in host_arrays.items()}
    flush = torch.empty(512 * 1024 * 1024 // 4, dtype=torch.float32, device="cuda")

    def flush_l2():
        flush.fill_(1.0)
        torch.cuda.synchronize()

    # launch shapes chosen by the library's autotuner on this instance (untimed)
    tune_main = compact_tuning(eng.autotune([inst], precision, [dev]))
    clocks = ClockSampler(local)     # started before the warm-up: sampling runs when timing starts
    clocks.start()
    for _ in range(args.warmup):
        eng.g0w0(inst, precision, device_arrays=dev)
    # ---------------- timed region: device events per solve
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    clocks.mark("begin")
    dev_ms, chi0_ms, launches, outs = [], [], 0, []
    for _ in range(args.steps):
        flush_l2()
        out = eng.g0w0(inst, precision, device_arrays=dev)
        st = eng.last_stats()
        dev_ms.append(out.device_ms)
        chi0_ms.append(st["stage_ms"][1])
        launches += st["kernel_launches"]
        outs.append(out)
    torch.cuda.synchronize()
    clocks.mark("end")
    if world > 1:
        dist.barrier()
    clk = clocks.stop()
    total_ms = float(sum(dev_ms))
    if world > 1:
        t = torch.tensor([total_ms], device="cuda", dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        total_ms = float(t.item())
    value = world * args.steps / (total_ms * 1e-3)
    stages = eng.last_stats()["stage_ms"]

    # ---------------- the other precision on the same instance (not part of `value`)
    other = RIGW_BF16X3 if precision == RIGW_FP64 else RIGW_FP64
    alt = None
    try:
        tune_alt = compact_tuning(eng.autotune([inst], other, [dev]))
        for _ in range(2):
            eng.g0w0(inst, other, device_arrays=dev)
        alt_ms, alt_chi0, alt_outs = [], [], []
        for _ in range(args.steps):
            flush_l2()
            o = eng.g0w0(inst, other, device_arrays=dev)
            alt_ms.append(o.device_ms)
            alt_chi0.append(eng.last_stats()["stage_ms"][1])
            alt_outs.append(o)
        alt = {"precision": "bf16x3" if other == RIGW_BF16X3 else "fp64",
               "value": args.steps / (sum(alt_ms) * 1e-3), "unit": "solves/s",
               "ms_per_step": float(np.mean(alt_ms)), "chi0_ms": float(np.mean(alt_chi0)),
               "stage_ms": eng.last_stats()["stage_ms"],
               "qp_diff_mev_vs_" + args.precision: float(
                   np.abs(alt_outs[-1].energy_qp_g - outs[-1].energy_qp_g).max() * HA_EV * 1e3),
               "tuning": tune_alt}
    except Exception as exc:    # precision unavailable on this device: reported, not hidden
        alt = {"error": str(exc)}

    # ---------------- end to end through the host-pointer C-ABI call
    pinned = {k: torch.from_numpy(np.ascontiguousarray(v)).pin_memory().numpy() for k, v in host_arrays.items()}
    inst_h = synth.GWInstance(**{**inst.__dict__})
    inst_h.m_ia = pinned["m_ia"]
    inst_h.m_sigma = pinned["m_pm"]
    h2d = sum(int(v.nbytes) for k, v in pinned.items() if k != "occ_sig")
    nreal = 2 * (inst.nomega_sigma // 2) + 1
    d2h = 8 * (2 + 2 * 2 * inst.nomega_sigma_calc + 2 * 2 * nreal + 3 * 2 + 4 * 2)
    for _ in range(2):
        eng.g0w0(inst_h, precision)
    if world > 1:
        dist.barrier()
    e2e_t = []
    for _ in range(args.steps):
        flush_l2()
        t0 = time.perf_counter()
        eng.g0w0(inst_h, precision)
        e2e_t.append(time.perf_counter() - t0)
    e2e_total = float(sum(e2e_t))
    if world > 1:
        t = torch.tensor([e2e_total], device="cuda", dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e2e_total = float(t.item())
    e2e_value = world * args.steps / e2e_total

    batched = None
    if args.batch_count > 0 and world == 1:
        try:
            batched = run_batched(eng, args.batch_count, args.batch_reps, flush_l2, args.batch_reps_fp64)
        except Exception as exc:    # reported, not hidden
            batched = {"error": str(exc)}
    ao_to_qp = h2o = contour = ri = None
    if world == 1:
        # the blocks below use their own contexts: release this one's plan arenas first
        eng.close()
        torch.cuda.empty_cache()
        try:
            ao_to_qp = run_ao_to_qp_block()
        except Exception as exc:    # reported, not hidden
            ao_to_qp = {"error": str(exc)}
        try:
            h2o = run_h2o_block()
        except Exception as exc:    # reported, not hidden
            h2o = {"error": str(exc)}
        try:
            contour = run_contour_block()
        except Exception as exc:    # reported, not hidden
            contour = {"error": str(exc)}
        try:
            ri = run_ri_block()
        except Exception as exc:    # reported, not hidden
            ri = {"error": str(exc)}
    sweep = None
    if args.sweep_block and world == 1:
        eng.close()
        torch.cuda.empty_cache()
        try:
            peaks0 = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
            sweep = run_sweep_block(measured_fp64_peak(torch), float(peaks0.get("bf16_tflops", 1590.0)))
        except Exception as exc:    # reported, not hidden
            sweep = {"error": str(exc)}
    serving = None
    if args.serving_window > 0 and world == 1:
        # the request loop sizes its worker arenas from free memory: release this
        # context's plan arenas and the batch inputs first
        eng.close()
        torch.cuda.empty_cache()
        try:
            serving = run_serving_block(args)
        except Exception as exc:    # reported, not hidden
            serving = {"error": str(exc)}

    if rank == 0:
        fp64_peak = measured_fp64_peak(torch)
        peaks = json.loads((ROOT / "MEASURED_PEAKS.json").read_text()) if (ROOT / "MEASURED_PEAKS.json").exists() else {}
        chi0_avg = float(np.mean(chi0_ms))
        # FP64 chi0: 34 exact int8 digit products per FP64 product; split precisions: theirs
        products = {"fp64": FP64_DIGIT_PRODUCTS, "bf16x3": 3}.get(args.precision, FP64_DIGIT_PRODUCTS)
        int8_peak = (1.0 if args.precision == "bf16x3" else 2.0) * float(peaks.get("bf16_tflops", 1590.0))
        achieved = products * chi0_flops(inst) / (chi0_avg * 1e-3) / 1e12
        traffic = profile_traffic("chi0_digits_naux840.txt" if products == FP64_DIGIT_PRODUCTS else
                                  "chi0_split_naux840.txt")
        roofline = {"kernel": "chi0 stage (row maxima, digits, digit_syrk_kernel<7>: 34 exact int8 digit products "
                              "of 55-bit operands on tcgen05, FP64 result)" if products == FP64_DIGIT_PRODUCTS else
                              "chi0 stage (split_bf16_kernel, split_syrk_kernel: 3 bf16 products on tcgen05)",
                    "bound": "tensor", "achieved": achieved, "peak": int8_peak, "unit": "TFLOP/s",
                    "frac": achieved / int8_peak, "traffic": traffic,
                    "peak_source": "MEASURED_PEAKS.json bf16_tflops (burst)" + (
                        "" if products == 3 else " x 2 (a cuBLAS rate doubled, not the int8 roof: "
                        "the product kernel alone runs at 3.5 Pop/s, 79% of the int8 pipe)"),
                    "algorithmic_flops_per_launch": chi0_flops(inst),
                    "fp64_tflops_algorithmic": chi0_flops(inst) / (chi0_avg * 1e-3) / 1e12,
                    "fp64_peak_measured_dgemm": fp64_peak,
                    "chi0_ms_per_launch": chi0_avg}
        line = {
            "metric": METRIC, "value": value, "unit": "solves/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64" if precision == RIGW_FP64 else "bf16x3+f64",
            "data": DATA,
            "config": bench_config(args.precision, world),
            "tuning": tune_main,
            "latency_ms": {"p50": float(np.percentile(dev_ms, 50)), "p99": float(np.percentile(dev_ms, 99))},
            "stage_ms": {"pack": stages[0], "chi0": stages[1], "eps_factor_solve": stages[2],
                         "sigma_qp": stages[3]},
            "achieved_tflops_solve": solve_flops(inst) / (total_ms / args.steps * 1e-3) / 1e12,
            "roofline": roofline,
            "e2e": {"value": e2e_value, "unit": "solves/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h},
            "gpu_launches": launches,
            "clocks": clk,
            "hbm_peak_gbs_measured": peaks.get("hbm_gbs"),
            "other_precision": alt,
            "batched": batched,
            "ao_to_qp": ao_to_qp,
            "h2o": h2o,
            "contour": contour,
            "ri_integrals": ri,
            "sweep": sweep,
            "serving": serving,
        }
        if alt and "chi0_ms" in alt and alt["precision"] == "bf16x3":
            # the tcgen05 kernel does 3 bf16 products of the chi0 contraction
            bf = peaks.get("bf16_tflops")
            ach = 3.0 * chi0_flops(inst) / (alt["chi0_ms"] * 1e-3) / 1e12
            alt["roofline_chi0"] = {"kernel": "split_bf16_kernel + split_syrk_kernel (tcgen05, 3 bf16 products)",
                                    "bound": "tensor", "achieved": ach, "peak": bf, "unit": "TFLOP/s",
                                    "frac": ach / bf if bf else None,
                                    "peak_source": "MEASURED_PEAKS.json bf16_tflops (burst, of measured)"}
            alt["speedup_vs_fp64"] = value / world / alt["value"] if precision == RIGW_BF16X3 else alt["value"] / (value / world)
        if world == 1 and not args.no_cpu_baseline:
            from threadpoolctl import threadpool_limits
            cores = os.cpu_count() or 1
            with threadpool_limits(limits=cores):
                t0 = time.perf_counter()
                ref = oracle_solve(inst)
                dt = time.perf_counter() - t0
            line["cpu_baseline"] = {"value": 1.0 / dt, "unit": "solves/s", "cores": cores, "kind": "port",
                                    "sample": "one full G0W0 solve of the same instance (CPU restatement of "
                                              "MOLGW's BLAS/LAPACK path, OpenBLAS threads)"}
            out = outs[-1]
            line["qp_error_mev_vs_oracle"] = float(np.abs(out.energy_qp_g - ref.energy_qp_g).max() * HA_EV * 1e3)
            line["homo_lumo_ev"] = [float(out.ehomo * HA_EV), float(out.elumo * HA_EV)]
            if h2o and "error" not in h2o:
                hinst, _ = h2o_instance()
                with threadpool_limits(limits=cores):
                    t0 = time.perf_counter()
                    for _ in range(5):
                        oracle_solve(hinst)
                    dt = (time.perf_counter() - t0) / 5
                h2o["cpu_baseline"] = {"value": 1.0 / dt, "unit": "solves/s", "cores": cores, "kind": "port",
                                       "sample": "five G0W0 solves of the H2O workload, CPU restatement"}
            if contour and "error" not in contour:
                from oracle import rigw_oracle as o
                (e_, occ_, m_ia_, m_sig_, smin, smax, nim, nre, nsg, stp, eta_) = contour_args(synth.single_instance_840())
                rng = o.selfenergy_set_state_range(e_.size, occ_, selfenergy_state_min=smin, selfenergy_state_max=smax)
                with threadpool_limits(limits=cores):
                    t0 = time.perf_counter()
                    ref_c = o.g0w0_contour(e_, occ_, m_ia_, m_sig_, rng, 0, nim, nre, nomega_sigma=nsg,
                                           step_sigma=stp, eta=eta_)
                    dt = time.perf_counter() - t0
                contour["cpu_baseline"] = {"value": 1.0 / dt, "unit": "solves/s", "cores": cores, "kind": "port",
                                           "sample": "one contour-deformation solve of the same instance, CPU "
                                                     "restatement (LAPACK DSYEV per frequency)"}
                contour["qp_error_mev_vs_oracle"] = float(
                    np.abs(np.array(contour["_qp"]) - ref_c.energy_qp_g).max() * HA_EV * 1e3)
            if ri and "error" not in ri:
                from oracle import gaussian_ri as gri
                sh, ax, _ = ri_cluster(2)
                to_g = lambda shells: [gri.Shell(x.am, x.alpha, x.coeff, x.center) for x in shells]
                bf_c, aux_c = gri.build_functions(to_g(sh)), gri.build_functions(to_g(ax))
                t0 = time.perf_counter()
                gri.coulomb_3center(bf_c, aux_c)
                dt = time.perf_counter() - t0
                gpu2 = ri["clusters"][0]["raw_3center_s"]
                ri["cpu_baseline"] = {"value": dt, "unit": "s", "cores": 1, "kind": "port",
                                      "sample": "(mu nu|P) of the 2-water cluster, the oracle's C McMurchie-Davidson "
                                                "integrals (one thread) with the pure transform",
                                      "gpu_s_same_sample": gpu2, "speedup": dt / gpu2}
        if isinstance(line.get("contour"), dict):
            line["contour"].pop("_qp", None)
        print(json.dumps(line), flush=True)
    eng.close()
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
