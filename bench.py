#!/usr/bin/env python
"""Benchmark of the FP8 block-scaled GEMM hot path (and, as extra keys, the MoE layer).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]

One "step" is one pass over the 18-shape benchmark sweep (M in {1024, 6144} x 9 (N,K) pairs, the
shape list of the reference's benchmark set).  `value` is total algorithmic FLOPs of a step divided
by the device time of a step, inputs resident in HBM.  `e2e` is the same sweep through the
`run` C-ABI entry with HOST operands: pinned host -> device copies of A, B and the scales and the
device -> host copy of C are inside the timed region.

With N > 1 (launched by torchrun, one rank per GPU) every rank runs the same sweep on its own GPU
(independent GEMMs: replicas only, weak scaling, no data-path collective); the step time is the
max over ranks.

`--impl reference` times the reference project's own PyTorch implementation of the path (`ref_kernel`,
scripts/problems/gemm/reference.py:40-85, unmodified, from oracle/_ref) on the host cores with every
thread the process may use, one pass over the same 18 shapes per step; where oracle/_ref is absent the
numpy restatement of it stands in and the line says so (`cpu_baseline.kind`).

The JSON line's `extras` hold the other configurations: the single-GPU MoE layer, the expert-parallel MoE
layer (all N ranks, strong scaling) and the N-split GEMM; the two sharded ones carry a `parity` block (every
rank checks rows of its result against the CPU oracle after the timed loop) and the run fails if one
misses.  Development aids: `--workload moe` (single-GPU
MoE layer alone), `--workload multi` (the `extras` alone, under torchrun for N > 1), `--ep-pull` (expert
outputs pulled by the combine instead of pushed by the second expert GEMM), `--shapes MxNxK,...`,
`--no-extras`, `--no-cpu-baseline`.
"""
import argparse
import ctypes
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

import numpy as np  # noqa: E402

NK_PAIRS = [(1536, 7168), (3072, 1536), (576, 7168), (7168, 256), (7168, 2048), (4608, 7168), (7168, 2304),
            (512, 7168), (4096, 512)]
SWEEP = [(m, n, k) for m in (1024, 6144) for (n, k) in NK_PAIRS]
# dram__bytes_read.sum + dram__bytes_write.sum of the GEMM kernel of each sweep shape, in SWEEP order, from one
# ncu pass (two DRAM counters, --clock-control none, caches flushed before each measured launch) over the fifth
# sweep of `bench.py --steps 2 --warmup 3 --no-cpu-baseline --no-extras`, taken with the kernels as they are now.
# Reads = A + B + scales once; C mostly stays in the 126 MB L2 at kernel end, hence traffic < algorithmic.  6144 x 4608 x
# 7168, whose operands and result do not fit the L2 together, reads its operands 1.6 times.
NCU_DRAM_BYTES = [18649600, 6407424, 11740416, 2171904, 16912640, 40669952, 19018496, 11280896, 2698240,
                  56980224, 14521856, 49644800, 30270208, 62302976, 155530496, 67401216, 49149696, 5478144]
# same two counters for the largest moe_gemm_kernel launch of the single-GPU MoE layer (fc1 of the routed experts and the
# shared one)
MOE_NCU_DRAM_BYTES = 2.99e9
# kernels of one layer through rf_moe_forward: router, top-k, sort, row gather, fc1, fc2, combine
MOE_LAYER_LAUNCHES = 7
METRIC = "fp8_blockscaled_gemm_tflops"
UNIT = "TFLOP/s"


def gemm_flops(m, n, k):
    return 2.0 * m * n * k


def gemm_bytes(m, n, k):
    """Algorithmic HBM bytes: fp8 operands and fp32 scales read once, bf16 C written once."""
    kb = k // 128
    nb = (n + 127) // 128
    return m * k + n * k + 4 * m * kb + 4 * nb * kb + 2 * m * n


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        try:
            p = json.load(open(path))
            return {"hbm_gbs": float(p["hbm_gbs"]), "bf16_tflops": float(p["bf16_tflops"]),
                    "bf16_tflops_sustained": float(p.get("bf16_tflops_sustained", p["bf16_tflops"])),
                    "source": "measured"}
        except Exception:
            pass
    return {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "bf16_tflops_sustained": 1400.0, "source": "fallback"}


# ----------------------------------------------------------------------------- clocks sampling --
class ClockSampler:
    """Samples SM clock and throttle reasons of one GPU while the timed region runs (read-only)."""

    def __init__(self, index: int):
        self.index = index
        self.samples = []
        self.reasons = set()
        self.max_mhz = None
        self._stop = threading.Event()
        self._thread = None
        self._nvml = None

    def start(self):
        try:
            import pynvml
            pynvml.nvmlInit()
            self._nvml = pynvml
            self._h = pynvml.nvmlDeviceGetHandleByIndex(self.index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self._h, pynvml.NVML_CLOCK_SM)
        except Exception:
            self._nvml = None
        self._thread = threading.Thread(target=self._loop, daemon=True)
        self._thread.start()

    def _loop(self):
        names = {
            0x8: "hw_slowdown", 0x40: "hw_thermal_slowdown", 0x20: "sw_thermal_slowdown", 0x4: "sw_power_cap",
            0x80: "hw_power_brake_slowdown", 0x2: "applications_clocks_setting",
        }
        while not self._stop.is_set():
            if self._nvml is not None:
                try:
                    n = self._nvml
                    self.samples.append(n.nvmlDeviceGetClockInfo(self._h, n.NVML_CLOCK_SM))
                    try:
                        r = n.nvmlDeviceGetCurrentClocksEventReasons(self._h)
                    except Exception:
                        r = n.nvmlDeviceGetCurrentClocksThrottleReasons(self._h)
                    for bit, name in names.items():
                        if r & bit:
                            self.reasons.add(name)
                except Exception:
                    pass
            else:
                try:
                    out = subprocess.run(
                        ["nvidia-smi", "-i", str(self.index), "--query-gpu=clocks.sm,clocks.max.sm,"
                         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
                         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap",
                         "--format=csv,noheader,nounits"], capture_output=True, text=True, timeout=5).stdout
                    f = [x.strip() for x in out.strip().split(",")]
                    self.samples.append(int(f[0]))
                    self.max_mhz = int(f[1])
                    for name, v in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"),
                                       f[2:6]):
                        if v.lower().startswith("active"):
                            self.reasons.add(name)
                except Exception:
                    pass
            self._stop.wait(0.004 if self._nvml is not None else 0.2)

    def stop(self):
        self._stop.set()
        if self._thread:
            self._thread.join(timeout=5)
        return {
            "sm_mhz": statistics.median(self.samples) if self.samples else None,
            "sm_max_mhz": self.max_mhz,
            "reasons": sorted(self.reasons),
            "samples": len(self.samples),
        }


# ------------------------------------------------------------------------------- CPU reference --
def sweep_config(world, shapes_arg=""):
    """The `config` object of the JSON line; both arms print the same one."""
    return {"workload": ("fp8 block-scaled GEMM, 18-shape sweep M in {1024,6144} x 9 (N,K)"
                         if not shapes_arg else "fp8 block-scaled GEMM, restricted to " + shapes_arg),
            "l2": "inputs larger than L2: one step touches ~1.0 GB; per-shape table rotates operand sets > L2",
            "launch": "one CUDA graph replay per step",
            "parallelism": "replicas" if world > 1 else "single"}


def host_threads():
    """Threads this process may use: every core of its affinity mask.  torchrun exports OMP_NUM_THREADS=1 to its
    workers, so the CPU arm sets its thread count itself instead of inheriting it."""
    try:
        return max(1, len(os.sched_getaffinity(0)))
    except AttributeError:
        return os.cpu_count() or 1


def load_reference_module():
    """The reference's scripts/problems/gemm/reference.py from oracle/_ref (written there by oracle/make_ref.py),
    imported the way scripts/eval.py:157-169 imports it.  None when the copy is not there."""
    base = os.path.join(ROOT, "oracle", "_ref", "scripts")
    prob = os.path.join(base, "problems", "gemm")
    if not os.path.exists(os.path.join(prob, "reference.py")) or not os.path.exists(os.path.join(base, "utils.py")):
        return None
    import importlib.util
    saved = list(sys.path)
    sys.path[:0] = [prob, base]
    try:
        spec = importlib.util.spec_from_file_location("task", os.path.join(prob, "task.py"))
        task = importlib.util.module_from_spec(spec)
        sys.modules["task"] = task
        spec.loader.exec_module(task)
        spec = importlib.util.spec_from_file_location("rf_reference_gemm", os.path.join(prob, "reference.py"))
        ref = importlib.util.module_from_spec(spec)
        spec.loader.exec_module(ref)
        return ref
    except Exception as e:                                  # an unreadable copy: say so and use the restatement
        print(f"bench.py: oracle/_ref could not be imported ({e}); using the numpy restatement", file=sys.stderr)
        return None
    finally:
        sys.path[:] = saved


class CpuArm:
    """The path on the host cores: the reference's own `ref_kernel` on CPU tensors (kind "reference") or, when
    oracle/_ref is absent, the numpy restatement of it (kind "port").  Same data recipe as the GPU arm."""

    def __init__(self, shapes):
        import torch
        from oracle import fp8_gemm as o
        self.threads = host_threads()
        torch.set_num_threads(self.threads)
        self.ref = load_reference_module()
        self.kind = "reference" if self.ref is not None else "port"
        self.shapes = list(shapes)
        self.problems = []
        for i, (m, n, k) in enumerate(self.shapes):
            a, b, a_s, b_s = o.generate_input(m, n, k, 100 + i, "baseline")
            if self.ref is not None:
                self.problems.append((torch.from_numpy(a).view(torch.float8_e4m3fn),
                                      torch.from_numpy(b).view(torch.float8_e4m3fn), torch.from_numpy(a_s),
                                      torch.from_numpy(b_s), torch.zeros((m, n), dtype=torch.bfloat16)))
            else:
                self.problems.append((a, b, a_s, b_s))
        self.flops = sum(gemm_flops(*x) for x in self.shapes)

    def one_pass(self, problems=None):
        """Seconds of one pass over the problems."""
        probs = self.problems if problems is None else problems
        t0 = time.perf_counter()
        if self.ref is not None:
            import torch
            with torch.no_grad():
                for data in probs:
                    self.ref.ref_kernel(data)
        else:
            from oracle import fp8_gemm as o
            from threadpoolctl import threadpool_limits
            with threadpool_limits(limits=self.threads):
                for (a, b, a_s, b_s) in probs:
                    o.fp8_gemm(a, b, a_s, b_s)
        return time.perf_counter() - t0

    def describe(self, passes, seconds):
        what = ("the reference's ref_kernel (scripts/problems/gemm/reference.py:40-85, unmodified, torch CPU)"
                if self.ref is not None else "numpy restatement of the reference's ref_kernel (oracle/_ref absent)")
        return (f"{passes} pass(es) of {what} over the {len(self.shapes)} shapes of the sweep "
                f"({self.flops / 1e9:.0f} GFLOP per pass, {seconds:.1f} s)")


def run_reference_arm(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    world = int(os.environ.get("WORLD_SIZE", "1"))
    arm = CpuArm(SWEEP)
    for _ in range(max(1, min(args.warmup, 1))):
        arm.one_pass(arm.problems[:2])
    steps = max(1, args.steps)
    times = [arm.one_pass() for _ in range(steps)]
    tsum = sum(times)
    val = arm.flops * steps / tsum / 1e12
    line = {
        "impl": "reference", "metric": METRIC, "value": val, "unit": UNIT, "n_gpus": args.gpus, "steps": steps,
        "warmup": args.warmup, "ms_per_step": tsum / steps * 1e3, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32 (CPU dequantised e4m3)", "data": "synthetic",
        "config": sweep_config(world, args.shapes),
        "cpu_baseline": {"value": val, "unit": UNIT, "cores": arm.threads, "kind": arm.kind,
                         "sample": arm.describe(steps, tsum)},
        "e2e": {"value": val, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)


# ------------------------------------------------------------------------- extra workloads --
def _timed(fn, iters, warm, dev, world, dist):
    """Device time per iteration (ms): CUDA events on the current stream, barrier + synchronize on
    both sides, max over ranks."""
    import torch
    for _ in range(warm):
        fn()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(iters):
        fn()
    e1.record()
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    t = torch.tensor([e0.elapsed_time(e1) / iters], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def moe_layer_flops(t, d, f, e, k):
    return 2.0 * t * d * e + 2.0 * t * k * 3 * d * f + 2.0 * t * 3 * d * f


def make_moe_weights(torch, dev, d, f, experts, seed, with_router_for=None):
    """Random-init weights with the reference generator's scales (scripts/problems/moe/reference.py:192-238),
    drawn on the device.  `experts` = list of local expert ids (names are local: experts.0...)."""
    g = torch.Generator(device=dev)
    w = {}
    g.manual_seed(seed)
    e_total = with_router_for
    w["router.weight"] = (torch.randn((e_total, d), device=dev, generator=g) / d ** 0.5).half()
    for j, shape, sc in ((0, (d, f), f), (1, (d, f), f), (2, (f, d), d)):
        w[f"shared_experts.{j}.weight"] = (torch.randn(shape, device=dev, generator=g) / sc ** 0.5).half()
    for j, e in enumerate(experts):
        g.manual_seed(seed * 1000 + e)
        w[f"experts.{j}.0.weight"] = (torch.randn((d, f), device=dev, generator=g) / f ** 0.5).half()
        w[f"experts.{j}.1.weight"] = (torch.randn((d, f), device=dev, generator=g) / f ** 0.5).half()
        w[f"experts.{j}.2.weight"] = (torch.randn((f, d), device=dev, generator=g) / d ** 0.5).half()
    return w


def measure_write_gbs(torch, dev):
    """Yardstick only: GB/s of a device memset over 1 GiB (best of 10).  HBM takes writes at about half the rate of
    the read+write copy the roofline's `peak` comes from, so a kernel whose traffic is mostly its bf16 result
    (the K <= 512 shapes) is bounded by this figure, not by the copy figure."""
    buf = torch.empty(1 << 30, dtype=torch.uint8, device=dev)
    for _ in range(3):
        buf.zero_()
    torch.cuda.synchronize()
    best = 0.0
    for _ in range(10):
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        buf.zero_()
        e1.record()
        torch.cuda.synchronize()
        best = max(best, buf.numel() / (e0.elapsed_time(e1) * 1e-3) / 1e9)
    del buf
    return best


def measure_fp8_peak(torch, dev):
    """Yardstick only: a plain (unscaled-block) FP8 GEMM of the vendor library, e4m3 8192^3 through
    torch._scaled_mm, best of 10 after warm-up, in TFLOP/s.  None when the call is not available."""
    try:
        n = 8192
        a = torch.randn((n, n), device=dev).to(torch.float8_e4m3fn)
        b = torch.randn((n, n), device=dev).to(torch.float8_e4m3fn).t()      # column-major second operand
        one = torch.ones((), device=dev)
        f = lambda: torch._scaled_mm(a, b, scale_a=one, scale_b=one, out_dtype=torch.bfloat16)
        for _ in range(3):
            f()
        torch.cuda.synchronize()
        best = 0.0
        for _ in range(10):
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record()
            f()
            e1.record()
            torch.cuda.synchronize()
            best = max(best, 2.0 * n ** 3 / (e0.elapsed_time(e1) * 1e-3) / 1e12)
        return best
    except Exception as e:
        print(f"bench.py: FP8 yardstick GEMM unavailable ({e})", file=sys.stderr)
        return None


def _all_ranks_ok(ok, dev, world, dist):
    import torch
    t = torch.tensor([1.0 if ok else 0.0], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MIN)
    return bool(t.item() > 0.5)


def check_nsplit_parity(torch, dist, dev, rank, world, a, a_s, c_full, m, n, kk, shard_seed):
    """Every rank: six full rows of its assembled C against the CPU oracle (every rank's B shard is regenerated
    from its seed), and a checksum of C that must agree on all ranks."""
    from oracle import fp8_gemm as og
    n_loc = n // world
    rows = [0, 1, m // 3, m // 2 + 5, m - 2, m - 1]
    ridx = torch.tensor(rows, device=dev)
    a_rows = a[ridx].view(torch.uint8).cpu().numpy()
    as_rows = a_s[ridx].cpu().numpy()
    got = c_full[ridx].view(torch.uint16).cpu().numpy()
    g = torch.Generator(device=dev)
    worst, bad = 0.0, 0
    for r in range(world):
        g.manual_seed(shard_seed + r)
        b_r = torch.randn((n_loc, kk), device=dev, generator=g).clamp_(-240, 240).to(torch.float8_e4m3fn)
        bs_r = ((0.5 + 1.5 * torch.rand((n_loc // 128, kk // 128), device=dev, generator=g)) * 2.0 ** -7).float()
        exp = og.fp8_gemm(a_rows, b_r.view(torch.uint8).cpu().numpy(), as_rows, bs_r.cpu().numpy())
        ok, nbad, mx = og.check(got[:, r * n_loc:(r + 1) * n_loc], exp)
        bad += int(nbad)
        worst = max(worst, float(mx))
        del b_r, bs_r
    # the same bytes everywhere: sum of C read as int16 (exact in int64), max and min over ranks must agree
    cs = c_full.view(torch.int16).to(torch.int64).sum().reshape(1)
    hi, lo = cs.clone(), cs.clone()
    if world > 1:
        dist.all_reduce(hi, op=dist.ReduceOp.MAX)
        dist.all_reduce(lo, op=dist.ReduceOp.MIN)
    same = bool((hi == lo).item())
    ok = _all_ranks_ok(bad == 0 and same, dev, world, dist)
    return {"ok": ok, "rows_checked_per_rank": len(rows), "elements_out_of_tolerance_rank0": bad,
            "max_abs_err_rank0": worst, "checksum_equal_on_all_ranks": same,
            "oracle": "oracle.fp8_gemm (restatement of scripts/problems/gemm/reference.py:40-87), rtol 2e-2 atol 1e-3"}


def check_ep_parity(torch, dist, dev, rank, world, layer, x, out, router_w_placed, bias_placed, order, d, f, e, k,
                    weight_seed):
    """Every rank: four of its tokens against the CPU oracle restricted to those tokens' experts.  Expert
    weights are seeded per ORIGINAL expert id, so any rank regenerates the few it needs; `order` maps a placed
    (renumbered) expert id to the original one."""
    from oracle import moe as om
    t_loc = x.shape[0]
    toks = [0, t_loc // 3, (2 * t_loc) // 3 + 1, t_loc - 1]
    tidx = torch.tensor(toks, device=dev)
    x_rows = x[tidx].cpu().numpy()
    logits_dev = layer.scores[tidx].cpu().numpy()
    idx_dev = layer.idx[tidx].cpu().numpy()
    out_dev = out[tidx].cpu().numpy()
    # router logits within tolerance of the oracle's; the top-k rule is then applied to the DEVICE logits
    ref_logits = om.router_logits(x_rows, router_w_placed.cpu().numpy(), bias_placed)
    ok_l, nb_l, mx_l = om.check(logits_dev, ref_logits)
    idx_ref, w_ref, _ = om.route(logits_dev, k)
    idx_exact = bool(np.array_equal(idx_ref, idx_dev))
    g = torch.Generator(device=dev)
    g.manual_seed(weight_seed)
    torch.randn((e, d), device=dev, generator=g)                   # the router draw precedes the shared expert's
    sh = [(torch.randn(shape, device=dev, generator=g) / sc ** 0.5).half().cpu().numpy()
          for shape, sc in (((d, f), f), ((d, f), f), ((f, d), d))]
    acc = om.linear_fp16(om.swiglu_fc1(x_rows, sh[0], sh[1]), sh[2]).astype(np.float32)
    cache = {}
    for ti in range(len(toks)):
        for j in range(k):
            orig = int(order[int(idx_ref[ti, j])])
            if orig not in cache:
                g.manual_seed(weight_seed * 1000 + orig)
                cache[orig] = [(torch.randn(shape, device=dev, generator=g) / sc ** 0.5).half().cpu().numpy()
                               for shape, sc in (((d, f), f), ((d, f), f), ((f, d), d))]
            wg, wu, wd = cache[orig]
            y = om.linear_fp16(om.swiglu_fc1(x_rows[ti:ti + 1], wg, wu), wd).astype(np.float32)
            acc[ti] += np.float32(w_ref[ti, j]) * y[0]
    ok_o, nb_o, mx_o = om.check(out_dev, acc.astype(np.float16))
    ok = _all_ranks_ok(bool(ok_l) and idx_exact and bool(ok_o), dev, world, dist)
    return {"ok": ok, "tokens_checked_per_rank": len(toks), "indices_exact_rank0": idx_exact,
            "logits_out_of_tolerance_rank0": int(nb_l), "output_out_of_tolerance_rank0": int(nb_o),
            "max_abs_err_rank0": float(mx_o),
            "oracle": "oracle.moe (restatement of scripts/problems/moe/reference.py:72-101), rtol 1e-2 atol 1e-2, "
                      "top-k indices exact on the device's logits"}


def run_extras(args, rank, world, dev, dist, peaks):
    """MoE layer tokens/s (single-GPU config and the expert-parallel config) and the N-split GEMM."""
    import torch
    from radeonflow_kernels_b200 import moe as M, multi_gpu as mg
    out = {}
    f16_peak = peaks["bf16_tflops"]

    # ---- config 3: single-GPU MoE layer, T=8192, d=7168, f=2048, E=32, top-4 (every rank runs a replica)
    d, f, e, k, t = 7168, 2048, 32, 4, 8192
    w = make_moe_weights(torch, dev, d, f, list(range(e)), 11, with_router_for=e)
    cfg = {"d_hidden": d, "d_expert": f, "n_routed_experts": e, "n_shared_experts": 1, "n_experts_per_token": k,
           "batch_size": 1, "seq_len": t}
    g = torch.Generator(device=dev)
    g.manual_seed(5)
    x = torch.randn((1, t, d), device=dev, dtype=torch.float16, generator=g)
    buf = M.MoEBuffers(x, w, cfg)
    L = _lib_handle()
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    ms = _timed(lambda: L.rf_moe_forward(ctypes.byref(buf.raw), None, sp, None), 10, 3, dev, world, dist)
    fl = moe_layer_flops(t, d, f, e, k)
    out["moe_single_gpu"] = {
        "config": "T=8192 d=7168 f=2048 E=32 top-4 + 1 shared, fp16, router GEMM included",
        "ms_per_layer": ms, "tokens_per_s": world * t / (ms * 1e-3), "tflops_per_gpu": fl / (ms * 1e-3) / 1e12,
        "frac_f16_peak": fl / (ms * 1e-3) / 1e12 / f16_peak, "parallelism": "replicas" if world > 1 else "single",
        "roofline": {"bound": "tensor", "achieved": fl / (ms * 1e-3) / 1e12, "peak": f16_peak, "unit": "TFLOP/s",
                     "frac": fl / (ms * 1e-3) / 1e12 / f16_peak,
                     "frac_of_sustained_peak": fl / (ms * 1e-3) / 1e12 / peaks["bf16_tflops_sustained"],
                     "kernel": "moe_gemm_kernel", "traffic": MOE_NCU_DRAM_BYTES,
                     "traffic_note": "DRAM bytes of the largest moe_gemm_kernel launch of the layer (fc1), ncu; "
                                     "algorithmic 2.69e9; achieved is layer FLOPs over layer time (all kernels)",
                     "peak_source": f"bf16_tflops of {peaks['source']} (the layer runs for milliseconds at the power "
                                    "cap: the sustained figure is the fairer one)"}}
    del buf, w, x
    torch.cuda.empty_cache()

    # ---- config 4: expert-parallel MoE, 32768 tokens in total, E=256 top-8, Zipf(1.1)-skewed routing
    d, f, e, k, t_total = 7168, 2048, 256, 8, 32768
    t_loc = t_total // world
    e_loc = e // world
    # Static load-aware placement decided before the timed region from a CALIBRATION batch drawn with another
    # seed than the timed batch: the router and top-k kernels give pairs per expert; experts are then renumbered
    # in placement order (router rows and bias permuted), which leaves the layer itself unchanged.
    # load skew: logit bias -1.1 * ln(1 + rank_e) with a seeded random rank per expert (Zipf(1.1) popularity)
    bias_np = (-1.1 * np.log1p(np.random.default_rng(17).permutation(e).astype(np.float64))).astype(np.float32)
    g.manual_seed(900 + rank)
    x_cal = torch.randn((t_loc, d), device=dev, dtype=torch.float16, generator=g)
    g.manual_seed(100 + rank)
    x = torch.randn((t_loc, d), device=dev, dtype=torch.float16, generator=g)
    g.manual_seed(13)
    router_w = (torch.randn((e, d), device=dev, generator=g) / d ** 0.5).half()
    cal_scores = torch.empty((t_loc, e), dtype=torch.float16, device=dev)
    cal_idx = torch.empty((t_loc, k), dtype=torch.int32, device=dev)
    cal_w = torch.empty((t_loc, k), dtype=torch.float16, device=dev)
    cal_src = torch.empty((t_loc * k,), dtype=torch.int32, device=dev)
    bias0 = torch.from_numpy(bias_np).to(dev)
    L.rf_moe_router_gemm(x_cal.data_ptr(), router_w.data_ptr(), bias0.data_ptr(), t_loc, e, d, cal_scores.data_ptr(),
                         sp)
    L.rf_moe_topk(cal_scores.data_ptr(), t_loc, e, k, cal_idx.data_ptr(), cal_w.data_ptr(), cal_src.data_ptr(), sp)
    loads = torch.bincount(cal_idx.reshape(-1).long(), minlength=e).double()
    if world > 1:
        dist.all_reduce(loads)
    order = mg.balanced_expert_placement(loads.cpu().numpy(), world)
    del x_cal, cal_scores, cal_idx, cal_w, cal_src
    w = make_moe_weights(torch, dev, d, f, [int(order[rank * e_loc + j]) for j in range(e_loc)], 13,
                         with_router_for=e)
    w["router.weight"] = router_w[torch.from_numpy(order).to(dev)].contiguous()
    cfg = {"d_hidden": d, "d_expert": f, "n_routed_experts": e, "n_shared_experts": 1, "n_experts_per_token": k,
           "batch_size": 1, "seq_len": t_loc}
    bias = torch.from_numpy(bias_np[order]).to(dev)
    layer = mg.ExpertParallelMoE(cfg, w, t_loc, dev, router_bias=bias, push_results=not args.ep_pull)
    if args.ep_dispatch_blocks:
        layer.set_dispatch_blocks(max(0, args.ep_dispatch_blocks))
    ms = _timed(lambda: layer.forward(x), 5, 2, dev, world, dist)
    layer.set_trace(True)
    y = layer.forward(x)
    stages = {name: round(ms_, 4) for name, ms_ in layer.stage_times_ms()}
    layer.set_trace(False)
    rows = torch.tensor([float(layer.received_rows())], dtype=torch.float64, device=dev)
    mx, sm = rows.clone(), rows.clone()
    if world > 1:
        dist.all_reduce(mx, op=dist.ReduceOp.MAX)
        dist.all_reduce(sm, op=dist.ReduceOp.SUM)
    parity = check_ep_parity(torch, dist, dev, rank, world, layer, x, y, w["router.weight"], bias_np[order], order, d,
                             f, e, k, 13)
    status = ctypes.c_int(0)
    L.rf_device_status(ctypes.byref(status))
    parity["device_status"] = status.value
    parity["ok"] = parity["ok"] and _all_ranks_ok(status.value == 0, dev, world, dist)
    fl = moe_layer_flops(t_total, d, f, e, k)
    peak_total = world * peaks["bf16_tflops_sustained"]
    nv = (world - 1) / world * t_loc * k * d * 2            # bytes each GPU sends (and receives) per direction
    bound_ms = max(fl / (peak_total * 1e12), 2 * nv / 770e9) * 1e3
    out["moe_expert_parallel"] = {
        "config": "32768 tokens, d=7168 f=2048 E=256 top-8 + 1 shared, Zipf(1.1) router bias; experts sharded E/N "
                  "per GPU by a static load-aware placement from a calibration batch drawn with another seed; "
                  "dispatch by peer stores, "
                  + ("combine by peer loads" if (args.ep_pull or world == 1) else
                     "expert outputs pushed home by the second GEMM's epilogue (peer stores), local combine"),
        "ms_per_layer": ms, "tokens_per_s": t_total / (ms * 1e-3), "tflops_total": fl / (ms * 1e-3) / 1e12,
        "stage_ms_rank0": stages, "scaling": "strong", "rows_per_gpu_max": mx.item(), "rows_per_gpu_mean": sm.item() / world,
        "imbalance_max_over_mean": mx.item() / (sm.item() / world), "parity": parity,
        "roofline": {"bound": "tensor", "achieved": fl / (ms * 1e-3) / 1e12, "peak": peak_total, "unit": "TFLOP/s",
                     "frac": fl / (ms * 1e-3) / 1e12 / peak_total, "kernel": "moe_gemm_kernel", "traffic": None,
                     "target_ms": bound_ms,
                     "peak_source": f"N x bf16_tflops_sustained of {peaks['source']}; target_ms = max(FLOPs / that, "
                                    "dispatch + return bytes per GPU / 770 GB/s measured peer bandwidth)"}}
    layer.close()
    del layer, w, x, y
    torch.cuda.empty_cache()
    if not parity["ok"]:
        raise SystemExit(f"bench.py: expert-parallel MoE parity failed on {world} GPU(s): {json.dumps(parity)}")

    # ---- config 2: M=16384 N=28672 K=7168 split along N, C assembled on every GPU by the epilogue
    m, n, kk = 16384, 28672, 7168
    n_loc = n // world
    g.manual_seed(7)
    a = torch.randn((m, kk), device=dev, generator=g).clamp_(-240, 240).to(torch.float8_e4m3fn)
    a_s = ((0.5 + 1.5 * torch.rand((m, kk // 128), device=dev, generator=g)) * 2.0 ** -7).float()
    g.manual_seed(70 + rank)
    b = torch.randn((n_loc, kk), device=dev, generator=g).clamp_(-240, 240).to(torch.float8_e4m3fn)
    b_s = ((0.5 + 1.5 * torch.rand((n_loc // 128, kk // 128), device=dev, generator=g)) * 2.0 ** -7).float()
    cbuf = mg.PeerBuffer(m * n * 2, dev)
    flag = torch.zeros(1, device=dev)

    def step():
        mg.fp8_gemm_nsplit(a, b, a_s, b_s, cbuf, m, n, kk)
        mg.stream_barrier(flag)
    ms = _timed(step, 5, 2, dev, world, dist)
    parity = check_nsplit_parity(torch, dist, dev, rank, world, a, a_s, cbuf.tensor(torch.bfloat16, (m, n)), m, n, kk,
                                 70)
    c_loc = torch.empty((m, n_loc), dtype=torch.bfloat16, device=dev)
    ms_local = _timed(lambda: L.rf_fp8_gemm(a.data_ptr(), b.data_ptr(), a_s.data_ptr(), b_s.data_ptr(),
                                            c_loc.data_ptr(), m, n_loc, kk, 1, None, 0, sp), 5, 2, dev, world, dist)
    fl = 2.0 * m * n * kk
    nv_bytes = (world - 1) / world * m * n * 2          # C bytes each GPU receives over NVLink
    fp8_peak = peaks.get("fp8_tflops") or 2 * peaks["bf16_tflops"]
    roof_ms = max(fl / world / (fp8_peak * 1e12), nv_bytes / 770e9) * 1e3
    out["gemm_nsplit"] = {
        "config": "M=16384 N=28672 K=7168 fp8, B row-partitioned, bf16 C all-gathered by epilogue peer stores",
        "ms": ms, "tflops_total": fl / (ms * 1e-3) / 1e12, "ms_gemm_only_local_c": ms_local,
        "tflops_total_gemm_only": fl / (ms_local * 1e-3) / 1e12, "scaling": "strong",
        "nvlink_bytes_in_per_gpu": nv_bytes, "roofline_ms": roof_ms, "parity": parity,
        "roofline": {"bound": "tensor" if fl / world / (fp8_peak * 1e12) > nv_bytes / 770e9 else "nvlink",
                     "achieved": roof_ms / ms, "peak": 1.0, "unit": "fraction of the target time", "frac": roof_ms / ms,
                     # (peer stores leave from the one-CTA tiles)
                     "kernel": "fp8_gemm_pair_kernel" if world == 1 else "fp8_gemm_kernel", "traffic": None,
                     "peak_source": "target time = max(FLOPs per GPU / FP8 peak of this run, C bytes received per GPU "
                                    "/ 770 GB/s measured peer bandwidth)"}}
    cbuf.close()
    if not parity["ok"]:
        raise SystemExit(f"bench.py: N-split GEMM parity failed on {world} GPU(s): {json.dumps(parity)}")
    return out


def run_moe_only(args):
    """Single-GPU MoE layer (config 3) alone: W warm-up layers, K timed layers, one JSON line."""
    import torch
    from radeonflow_kernels_b200 import moe as M, build
    torch.cuda.set_device(0)
    dev = torch.device("cuda", 0)
    build.build()
    L = _lib_handle()
    d, f, e, k, t = 7168, 2048, 32, 4, 8192
    w = make_moe_weights(torch, dev, d, f, list(range(e)), 11, with_router_for=e)
    cfg = {"d_hidden": d, "d_expert": f, "n_routed_experts": e, "n_shared_experts": 1, "n_experts_per_token": k,
           "batch_size": 1, "seq_len": t}
    g = torch.Generator(device=dev)
    g.manual_seed(5)
    x = torch.randn((1, t, d), device=dev, dtype=torch.float16, generator=g)
    buf = M.MoEBuffers(x, w, cfg)
    sp = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    steps = min(args.steps, 50)
    ms = _timed(lambda: L.rf_moe_forward(ctypes.byref(buf.raw), None, sp, None), steps, max(3, args.warmup), dev, 1,
                None)
    fl = moe_layer_flops(t, d, f, e, k)
    peaks = measured_peaks()
    print(json.dumps({
        "metric": "moe_layer_tokens_per_s", "value": t / (ms * 1e-3), "unit": "tokens/s", "n_gpus": 1, "steps": steps,
        "warmup": max(3, args.warmup), "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "fp16 x fp16 -> f32", "data": "synthetic",
        "config": {"workload": "MoE layer T=8192 d=7168 f=2048 E=32 top-4 + 1 shared (weights 3 GB > L2)"},
        "roofline": {"bound": "tensor", "achieved": fl / (ms * 1e-3) / 1e12, "peak": peaks["bf16_tflops"],
                     "unit": "TFLOP/s", "frac": fl / (ms * 1e-3) / 1e12 / peaks["bf16_tflops"],
                     "traffic": MOE_NCU_DRAM_BYTES,
                     "traffic_note": "DRAM bytes of the largest moe_gemm_kernel launch (fc1), ncu capture; "
                                     "algorithmic 2.69e9; achieved/frac are layer FLOPs over layer time (all "
                                     "kernels of the layer)",
                     "kernel": "moe_gemm_kernel"},
        "gpu_launches": MOE_LAYER_LAUNCHES * steps}), flush=True)


def run_multi_gpu_only(args):
    """The multi-GPU workloads alone (expert-parallel MoE, N-split GEMM; plus the single-GPU MoE replica):
    one JSON line with the `extras` object of the full run.  Launch under torchrun for N > 1."""
    import torch
    import torch.distributed as dist
    from radeonflow_kernels_b200 import build
    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
    build.build()
    extras = run_extras(args, rank, world, dev, dist, measured_peaks())
    if rank == 0:
        print(json.dumps({"workload": "multi-gpu extras", "n_gpus": world, "extras": extras}), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


def _lib_handle():
    from radeonflow_kernels_b200 import _lib
    return _lib.lib()

# ------------------------------------------------------------------------------------ GPU arm --
def run_gpu_arm(args):
    import torch
    import torch.distributed as dist

    from radeonflow_kernels_b200 import _lib, build

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if not torch.cuda.is_available():
        raise SystemExit("bench.py: no CUDA device; the GPU arm has no CPU fallback")
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
    build.build()
    L = _lib.lib()
    stream = torch.cuda.current_stream()
    sptr = ctypes.c_void_p(stream.cuda_stream)

    # ---- resident operands, one set per shape (the sweep touches ~1 GB per step, > 126 MB L2)
    rng = np.random.default_rng(1234 + rank)
    shapes = []
    for i, (m, n, k) in enumerate(SWEEP):
        # device-side generation keeps set-up short: random e4m3 bytes with |x| <= 240 drawn from N(0,1)
        g = torch.Generator(device=dev)
        g.manual_seed(1000 + i)
        a = torch.randn((m, k), device=dev, generator=g).clamp_(-240, 240).to(torch.float8_e4m3fn)
        b = torch.randn((n, k), device=dev, generator=g).clamp_(-240, 240).to(torch.float8_e4m3fn)
        kb, nb = k // 128, (n + 127) // 128
        a_s = ((0.5 + 1.5 * torch.rand((m, kb), device=dev, generator=g)) * 2.0 ** -7).float()
        b_s = ((0.5 + 1.5 * torch.rand((nb, kb), device=dev, generator=g)) * 2.0 ** -7).float()
        c = torch.empty((m, n), dtype=torch.bfloat16, device=dev)
        shapes.append({"m": m, "n": n, "k": k, "a": a, "b": b, "as": a_s, "bs": b_s, "c": c})
    del rng

    def launch(s):
        # `sptr` is rebound to the capturing stream while a graph is recorded
        L.run(s["a"].data_ptr(), s["b"].data_ptr(), s["as"].data_ptr(), s["bs"].data_ptr(), s["c"].data_ptr(),
              s["m"], s["n"], s["k"], None, sptr)

    def sweep():
        for s in shapes:
            launch(s)

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    launches_per_step = 0
    for s in shapes:
        sp = L.rf_fp8_gemm_choose_split(s["m"], s["n"], s["k"])
        s["split"] = sp
        launches_per_step += L.rf_fp8_gemm_kernel_launches(s["m"], s["n"], s["k"])

    for _ in range(max(3, args.warmup)):
        sweep()
    barrier()

    # The sweep is launch-bound on its small shapes, so one step is captured as a CUDA graph (18 GEMM
    # launches plus the split-K fix-ups) and a step is one replay.  Capture runs on a side stream.
    cap_stream = torch.cuda.Stream(device=dev)
    sptr_main = sptr
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(cap_stream):
        sptr = ctypes.c_void_p(cap_stream.cuda_stream)
        with torch.cuda.graph(graph, stream=cap_stream):
            sweep()
    sptr = sptr_main
    for _ in range(max(3, args.warmup)):
        graph.replay()
    barrier()

    sampler = ClockSampler(local_rank)
    sampler.start()
    e0 = torch.cuda.Event(enable_timing=True)
    e1 = torch.cuda.Event(enable_timing=True)
    barrier()
    e0.record(stream)
    for _ in range(args.steps):
        graph.replay()
    e1.record(stream)
    barrier()
    ms_total = e0.elapsed_time(e1)
    clocks = sampler.stop()

    t = torch.tensor([ms_total], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms_step = float(t.item()) / args.steps
    step_flops = sum(gemm_flops(*x) for x in SWEEP)
    value = world * step_flops / (ms_step * 1e-3) / 1e12

    # ---- per-shape table: each shape alone, as a graph of R launches that rotate over R operand sets
    # whose total footprint exceeds L2 (so every launch reads its operands from HBM)
    peaks = measured_peaks()
    # FP8 tensor peak: measured in this run with a plain vendor-library FP8 GEMM (a yardstick, not part of the
    # path); 2 x the measured bf16 figure only if that call is unavailable
    fp8_measured = measure_fp8_peak(torch, dev)
    fp8_assumed = 2.0 * peaks["bf16_tflops"]
    fp8_peak = fp8_measured if fp8_measured else fp8_assumed
    peaks["fp8_tflops"] = fp8_peak
    write_gbs = measure_write_gbs(torch, dev)
    per_shape = []
    for s in shapes:
        m, n, k = s["m"], s["n"], s["k"]
        foot = gemm_bytes(m, n, k)
        reps = int(min(24, max(2, -(-300e6 // foot))))
        sets = [s]
        for _ in range(reps - 1):
            sets.append({"m": m, "n": n, "k": k, "a": s["a"].clone(), "b": s["b"].clone(), "as": s["as"].clone(),
                         "bs": s["bs"].clone(), "c": torch.empty_like(s["c"])})
        g2 = torch.cuda.CUDAGraph()
        with torch.cuda.stream(cap_stream):
            sptr = ctypes.c_void_p(cap_stream.cuda_stream)
            with torch.cuda.graph(g2, stream=cap_stream):
                for x in sets:
                    launch(x)
        sptr = sptr_main
        g2.replay()
        torch.cuda.synchronize()
        ts = []
        for _ in range(5):
            a0 = torch.cuda.Event(enable_timing=True)
            a1 = torch.cuda.Event(enable_timing=True)
            a0.record(stream)
            g2.replay()
            a1.record(stream)
            torch.cuda.synchronize()
            ts.append(a0.elapsed_time(a1) * 1e3 / reps)
        us = min(ts)
        fl, by = gemm_flops(m, n, k), float(foot)
        per_shape.append({
            "m": m, "n": n, "k": k, "split_k": s["split"], "us": round(us, 2),
            "tflops": round(fl / us / 1e6, 1), "frac_fp8_peak": round(fl / us / 1e6 / fp8_peak, 3),
            "gbs": round(by / us / 1e3, 1), "frac_hbm": round(by / us / 1e3 / peaks["hbm_gbs"], 3),
            # the shape's own bound: the slower of its tensor time and its HBM time, over the measured time
            "frac_of_bound": round(max(fl / (fp8_peak * 1e6), by / (peaks["hbm_gbs"] * 1e3)) / us, 3),
            # the same with the result's write time at the measured write-only rate as a third bound
            "frac_of_bound_with_write": round(max(fl / (fp8_peak * 1e6), by / (peaks["hbm_gbs"] * 1e3),
                                                  2.0 * m * n / (write_gbs * 1e3)) / us, 3),
            "rotating_sets": reps,
        })
        del sets, g2
    status = ctypes.c_int(0)
    L.rf_device_status(ctypes.byref(status))
    if status.value != 0:
        raise SystemExit(f"bench.py: device status {status.value}: a bounded wait expired; numbers are invalid")

    # ---- end to end through `run` with host operands (pinned), copies inside the timed region
    host = []
    h2d = d2h = 0
    for s in shapes:
        h = {k2: s[k2].cpu().pin_memory() for k2 in ("a", "b", "as", "bs")}
        h["c"] = torch.empty(s["c"].shape, dtype=torch.bfloat16).pin_memory()
        host.append(h)
        h2d += sum(h[k2].numel() * h[k2].element_size() for k2 in ("a", "b", "as", "bs"))
        d2h += h["c"].numel() * 2

    # Three streams, as a host application would drive `run`: operands go up on one stream, the GEMMs run
    # on the second, results come back on the third; events chain shape i's copy-in -> GEMM -> copy-out,
    # so PCIe traffic in both directions overlaps the compute of neighbouring shapes.
    s_in = torch.cuda.Stream(device=dev)
    s_out = torch.cuda.Stream(device=dev)
    ev_in = [torch.cuda.Event() for _ in shapes]
    ev_mm = [torch.cuda.Event() for _ in shapes]
    ev_out = [torch.cuda.Event() for _ in shapes]

    def e2e_step():
        for i, (s, h) in enumerate(zip(shapes, host)):
            with torch.cuda.stream(s_in):
                s_in.wait_event(ev_mm[i])              # the previous step's GEMM has consumed the operands
                for k2 in ("a", "b", "as", "bs"):
                    s[k2].copy_(h[k2], non_blocking=True)
                ev_in[i].record(s_in)
            stream.wait_event(ev_in[i])
            stream.wait_event(ev_out[i])               # the previous step's read-back of C is done
            launch(s)
            ev_mm[i].record(stream)
            with torch.cuda.stream(s_out):
                s_out.wait_event(ev_mm[i])
                h["c"].copy_(s["c"], non_blocking=True)
                ev_out[i].record(s_out)
        stream.wait_stream(s_out)                      # the step ends when its last result is on the host

    e2e_steps = max(1, min(args.steps, 5))
    e2e_step()
    barrier()
    f0 = torch.cuda.Event(enable_timing=True)
    f1 = torch.cuda.Event(enable_timing=True)
    f0.record(stream)
    for _ in range(e2e_steps):
        e2e_step()
    f1.record(stream)
    barrier()
    t2 = torch.tensor([f0.elapsed_time(f1)], dtype=torch.float64, device=dev)
    if world > 1:
        dist.all_reduce(t2, op=dist.ReduceOp.MAX)
    e2e_ms = float(t2.item()) / e2e_steps
    e2e_val = world * step_flops / (e2e_ms * 1e-3) / 1e12

    extras = None
    if not args.no_extras:
        del host
        torch.cuda.empty_cache()
        extras = run_extras(args, rank, world, dev, dist, peaks)

    if rank == 0:
        cpu = None
        if world == 1 and not args.no_cpu_baseline:
            # bounded sample of the same workload on the host cores: whole passes over the 18 shapes until
            # about 12 s of CPU work have been timed (at least two passes after one warm-up of two shapes)
            arm = CpuArm(SWEEP)
            arm.one_pass(arm.problems[:2])
            tsec, reps = 0.0, 0
            while reps < 2 or (tsec < 12.0 and reps < 20):
                tsec += arm.one_pass()
                reps += 1
            cpu = {"value": arm.flops * reps / tsec / 1e12, "unit": UNIT, "cores": arm.threads, "kind": arm.kind,
                   "sample": arm.describe(reps, tsec)}
        achieved = step_flops / (ms_step * 1e-3) / 1e12
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": max(3, args.warmup), "ms_per_step": ms_step, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "fp8 e4m3 x e4m3 -> f32 (exact f32 block scales), bf16 out",
            "data": "synthetic",
            "config": sweep_config(world, args.shapes),
            "roofline": {"bound": "tensor", "achieved": achieved, "peak": fp8_peak, "unit": "TFLOP/s",
                         "frac": achieved / fp8_peak,
                         "frac_of_2x_bf16_burst": achieved / fp8_assumed,
                         "frac_of_2x_bf16_sustained": achieved / (2.0 * peaks["bf16_tflops_sustained"]),
                         "traffic": (sum(NCU_DRAM_BYTES) / len(NCU_DRAM_BYTES) if not args.shapes else None),
                         "traffic_note": "DRAM bytes per GEMM launch (10 of the 18 shapes run fp8_gemm_pair_kernel, 8 "
                                         "fp8_gemm_kernel), mean over the 18 shapes, from an ncu capture "
                                         "of one whole sweep after the warm-up sweeps (caches flushed per launch); "
                                         f"algorithmic mean {sum(gemm_bytes(*x) for x in SWEEP) / len(SWEEP):.0f}",
                         "peak_source": ("plain FP8 GEMM of the vendor library (torch._scaled_mm, e4m3 8192^3, best of 10) "
                                         "measured in this run as a yardstick" if fp8_measured else
                                         f"2 x bf16_tflops of {peaks['source']} (FP8 yardstick GEMM unavailable)"),
                         "peak_2x_bf16_burst": fp8_assumed,
                         "hbm_write_only_gbs": round(write_gbs, 1),
                         "hbm_write_only_note": "device memset of 1 GiB measured in this run; the third bound of the "
                                                "per-shape frac_of_bound_with_write (result bytes / this rate)",
                         "kernel": "fp8_gemm_pair_kernel"},
            "cpu_baseline": cpu,
            "e2e": {"value": e2e_val, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                    "ms_per_step": e2e_ms},
            "gpu_launches": launches_per_step * args.steps,
            "clocks": clocks,
            "shapes": per_shape,
            "extras": extras,
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=None)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-extras", action="store_true", help="skip the MoE and N-split GEMM workloads")
    ap.add_argument("--ep-dispatch-blocks", type=int, default=0,
                    help="expert-parallel MoE: SMs the dispatch owns (0 = library default: 32 on 2 to 4 GPUs; "
                         "-1 = none, the dispatch spreads over every SM)")
    ap.add_argument("--ep-pull", action="store_true",
                    help="expert-parallel MoE: combine pulls the expert outputs instead of fc2 pushing them")
    ap.add_argument("--workload", default="sweep", choices=["sweep", "moe", "multi"],
                    help="sweep = the FP8 GEMM benchmark line (default); moe = only the single-GPU MoE layer "
                         "(profiling aid: prints its own line, metric moe_layer_tokens_per_s)")
    ap.add_argument("--shapes", default="", help="restrict the sweep, e.g. 6144x4608x7168,1024x512x7168 "
                                                 "(profiling aid; the JSON line names the restricted workload)")
    args = ap.parse_args()
    if args.steps is None:
        args.steps = 200 if args.impl == "b200" else 10
    if args.shapes:
        args.no_extras = True
        global SWEEP
        SWEEP = [tuple(int(v) for v in t.split("x")) for t in args.shapes.split(",")]
    if args.impl == "reference":
        run_reference_arm(args)
    elif args.workload == "moe":
        run_moe_only(args)
    elif args.workload == "multi":
        run_multi_gpu_only(args)
    else:
        run_gpu_arm(args)


if __name__ == "__main__":
    main()
