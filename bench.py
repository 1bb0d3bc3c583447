#!/usr/bin/env python
"""Benchmark of the GEMM hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Workload (all N): the M-sharded bf16 GEMM M=32768, N=K=8192 (fp32 accumulate, bf16 out). Inputs follow the
seeded recipe of the parity tests: one CPU generator with seed 0 draws A (normal(0,1)/sqrt(K)) and then B, both
cast to bf16, so every machine and every rank sees the same bytes; rank r of N takes rows
[r*M/N, (r+1)*M/N) of A against a replicated B; no data-path collective. Total work is fixed, so scaling is
"strong"; at N=1 one GPU computes the whole product. A "step" is one pass of the rank's slab through the
tcgen05 kernel.

Outside the timed region every rank checks its result against the CPU oracle (``oracle_check``): eight random
128-row blocks of its slab at every N, and every row at N=1; a failed check ends the run with a non-zero exit
code. At N=1 a second JSON line, on stderr, carries under ``other_workloads`` the other single-GPU configs - fp32 1024^3 and
4096^3 (fp16 parts and FFMA SIMT), bf16 8192^3 and the rectangular sweep M in {128, 512, 2048} x N, K in {4096, 11008}
x {fp32, bf16} (24 points) - each with its roofline and the same shape through cuBLAS (``torch.matmul`` on the device) timed
the same way, and the operators around the product (batched, strided, the attention-shaped chain as three launches
and as one fused kernel), each beside its PyTorch library call and checked against the host composition at fp32.

Prints ONE JSON line on rank 0's stdout (metric: GEMM TFLOP/s, device-timed with CUDA events, max over ranks), of a few
KB: readers that keep the end of the output keep all of it.
``--impl reference`` times the reference's CPU path for the same metric: ``torch.matmul`` on host tensors (the
reference's own correctness oracle, Runtime/python/kcg/KCGTask.py:94) with all host threads, operands built
once before the clock starts, only the call between the two timestamps (KCGTask.py:124-130).
"""
import argparse
import json
import math
import os
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

M_TOTAL, N_SIZE, K_SIZE = 32768, 8192, 8192
METRIC = "GEMM TFLOP/s (device-timed) bf16 32768x8192x8192 M-sharded, fp32 accumulate"
UNIT = "TFLOP/s"
TOL_16BIT, TOL_FP32 = 2e-2, 1e-4  # max |c - ref| / max(|ref|, rms(ref)): bf16/fp16 vs fp32 accumulation, fp32 vs fp64
L2_BYTES = 126e6


def env_int(name, default):
    try:
        return int(os.environ.get(name, default))
    except ValueError:
        return default


def measured_peaks():
    from codegendemo_b200.kcg import roofline as rl
    return rl.load_peaks(os.path.join(ROOT, "MEASURED_PEAKS.json"))


def seeded_operands(M, N, K, torch_dtype, dist, seed=0):
    """A (M x K) then B (K x N) from one CPU generator: uniform[-1, 1) or normal(0,1)/sqrt(K), cast afterwards.
    The same recipe as the parity tests' inputs; identical bytes on every machine."""
    import torch
    g = torch.Generator().manual_seed(seed)
    if dist == "uniform":
        A = torch.rand(M, K, generator=g) * 2 - 1
        B = torch.rand(K, N, generator=g) * 2 - 1
    else:
        A = torch.randn(M, K, generator=g) / math.sqrt(K)
        B = torch.randn(K, N, generator=g) / math.sqrt(K)
    return A.to(torch_dtype), B.to(torch_dtype)


class ClockSampler:
    """Samples SM clock, power and throttle reasons with nvidia-smi while the GPU works.

    Each sample carries nvidia-smi's own timestamp, so `window()` can keep the samples that fall inside a
    timed region; when that region is too short for three samples `stop()` widens the window to the warm-up
    launches that run right before it (same kernel, same load) and the result says so.
    """
    QUERY = ("timestamp,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    NAMES = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.proc = None
        self.lines = []
        self.thread = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits", "-lms", "20",
                 "-i", str(self.gpu)], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
            return
        self.thread = threading.Thread(target=self._pump, daemon=True)
        self.thread.start()

    def _pump(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    @staticmethod
    def _epoch(stamp: str):
        import datetime
        try:
            return datetime.datetime.strptime(stamp.strip(), "%Y/%m/%d %H:%M:%S.%f").timestamp()
        except ValueError:
            return None

    def samples(self):
        out = []
        for ln in list(self.lines):
            parts = [p.strip() for p in ln.split(",")]
            if len(parts) < 9:
                continue
            try:
                rec = {"t": self._epoch(parts[0]), "sm": float(parts[1]), "max": float(parts[2]),
                       "power": float(parts[3])}
            except ValueError:
                continue
            rec["reasons"] = [n for n, v in zip(self.NAMES, parts[5:9]) if v.lower().startswith("active")]
            out.append(rec)
        return out

    @staticmethod
    def summarise(used, label):
        sm = sorted(r["sm"] for r in used)
        return {"sm_mhz": sm[len(sm) // 2] if sm else None,
                "sm_max_mhz": max((r["max"] for r in used), default=None),
                "power_w_max": max((r["power"] for r in used), default=None),
                "samples": len(used), "window": label,
                "reasons": sorted({x for r in used for x in r["reasons"]})}

    def window(self, lo, hi, label):
        """Summary of the samples taken between two host timestamps (the sampler keeps running)."""
        used = [r for r in self.samples() if r["t"] is not None and lo <= r["t"] <= hi]
        return self.summarise(used, label)

    def stop(self, timed=(None, None), loaded=(None, None)) -> dict:
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        samples = self.samples()

        def window(lo, hi):
            if lo is None:
                return []
            return [r for r in samples if r["t"] is not None and lo <= r["t"] <= hi]

        used, label = window(*timed), "timed region"
        if len(used) < 3:
            used, label = window(*loaded), "warm-up + timed region"
        if len(used) < 1:
            used, label = samples, "whole run"
        return self.summarise(used, label)


def build_bf16_kernel(m_rows: int, device: int):
    from codegendemo_b200.kcg.matmul_op import build_kernel, tuned_config
    from codegendemo_b200.kcg.Utils import EnumKernelDType as E
    kpm = tuned_config(m_rows, N_SIZE, K_SIZE, E.bfloat16)  # kernel database entry, else the B200 rule of thumb
    return kpm, build_kernel(kpm, device)


# ------------------------------------------------------------------------------------ oracle check
def rel_error(c, ref):
    """max |c - ref| / max(|ref|, rms(ref)) on host tensors (the gate of the parity tests), and a NaN flag."""
    import torch
    c, ref = c.double(), ref.double()
    if torch.isnan(c).any().item():
        return float("inf"), True
    rms = ref.pow(2).mean().sqrt().clamp_min(1e-300)
    return float(((c - ref).abs() / torch.maximum(ref.abs(), rms)).max().item()), False


def oracle_check(c_dev, A_slab, B, full: bool, blocks: int = 8, seed: int = 0):
    """This rank's device result against the CPU oracle (``oracle.host_matmul``: the reference's ``torch.matmul``
    check on host tensors, fp32 accumulation for bf16 data), outside any timed region: `blocks` random 128-row
    blocks of the slab, and every row when `full`. Test infrastructure used as the checker only."""
    import torch
    from oracle import oracle
    rows = A_slab.shape[0]
    nb = rows // 128
    g = torch.Generator().manual_seed(1000 + seed)
    pick = torch.randperm(nb, generator=g)[:min(blocks, nb)].sort().values.tolist()
    worst, nan = 0.0, False
    for b in pick:
        ref = oracle.host_matmul(A_slab[b * 128:(b + 1) * 128], B)
        e, n = rel_error(c_dev[b * 128:(b + 1) * 128].cpu().float(), ref)
        worst, nan = max(worst, e), nan or n
    out = {"blocks": len(pick), "block_rows": 128, "max_rel": worst}
    if full:
        t0 = time.perf_counter()
        worst_full = 0.0
        chunk = 4096
        for r0 in range(0, rows, chunk):
            ref = oracle.host_matmul(A_slab[r0:r0 + chunk], B)
            e, n = rel_error(c_dev[r0:r0 + chunk].cpu().float(), ref)
            worst_full, nan = max(worst_full, e), nan or n
        out.update({"full_rows": rows, "full_max_rel": worst_full, "full_check_s": round(time.perf_counter() - t0, 1)})
        worst = max(worst, worst_full)
    out.update({"tol": TOL_16BIT, "ok": bool(worst <= TOL_16BIT and not nan),
                "against": "oracle.host_matmul (torch.matmul on host tensors, fp32 accumulation)"})
    return out


# ------------------------------------------------------------------------------------ timing helpers
def time_launches(fn, launches, warmup):
    """Per-launch device times (ms): CUDA events on the launching stream around every launch, launches queued
    back to back (no host synchronisation in between)."""
    import torch
    for _ in range(warmup):
        fn()
    torch.cuda.synchronize()
    evs = [torch.cuda.Event(enable_timing=True) for _ in range(launches + 1)]
    evs[0].record()
    for i in range(launches):
        fn()
        evs[i + 1].record()
    torch.cuda.synchronize()
    return [evs[i].elapsed_time(evs[i + 1]) for i in range(launches)]


def time_graph(fn, launches, replays=5):
    """Mean device time per launch (ms) when `launches` launches are replayed from a CUDA graph: no host work
    between kernels, so it shows what the GPU alone needs - for kernels of a few microseconds the event-timed
    figure above is bounded by the host's launch rate instead. None when the capture is not possible."""
    import torch
    try:
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            for _ in range(3):
                fn()  # the library sets up this stream's status block and workspace outside the capture
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            for _ in range(launches):
                fn()
        graph.replay()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(replays):
            graph.replay()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1) / (replays * launches)
    except Exception:  # an extra figure: never lose the line over it
        torch.cuda.synchronize()
        return None


def other_workloads(device: int, peaks: dict, sampler: "ClockSampler", launches: int = 20):
    """Device-timed figures for the remaining single-GPU configs. Per workload: our kernel (the config the
    operator picks) and cuBLAS (``torch.matmul`` on the device, a comparison) timed the same way - median of
    `launches` back-to-back launches; the roofline min(tensor peak, arithmetic intensity x measured HBM bandwidth);
    the largest difference between the two results. Problems that fit the L2 rotate over copies of their operands
    so that every launch starts cold. One clock sample per group of workloads."""
    import torch
    from codegendemo_b200._lib import KERNEL_F32_SPLIT
    from codegendemo_b200.kcg import roofline as rl
    from codegendemo_b200.kcg.matmul_op import build_kernel, default_config, tuned_config
    from codegendemo_b200.kcg.Utils import EnumKernelDType as E
    simt = dict(KERNEL_VARIANT=1, BLOCK_SIZE_M=128, BLOCK_SIZE_N=128, BLOCK_SIZE_K=16, THREAD_SIZE_M=8,
                THREAD_SIZE_N=8, BLOCK_LAYOUT_M=4, BLOCK_LAYOUT_N=2, WARP_LAYOUT_M=4, WARP_LAYOUT_N=8,
                WARP_SCATTER_WIDTH_A=4, WARP_SCATTER_WIDTH_B=4, THREAD_SCATTER_WIDTH_A=4, THREAD_SCATTER_WIDTH_B=4)
    f32, bf16 = (E.float32, torch.float32), (E.bfloat16, torch.bfloat16)
    groups = [
        ("square fp32", [("c1 fp32 1024^3 3xTF32", 1024, 1024, 1024, f32, "uniform", None),
                         ("c2 fp32 4096^3 fp16 parts", 4096, 4096, 4096, f32, "uniform", None),
                         ("c2 fp32 4096^3 FFMA SIMT", 4096, 4096, 4096, f32, "uniform", simt)]),
        ("square bf16", [("c3 bf16 8192^3", 8192, 8192, 8192, bf16, "normal", None)]),
    ]
    for n in (4096, 11008):
        for k in (4096, 11008):
            for (edt, tdt), tag in ((bf16, "bf16"), (f32, "fp32")):
                groups.append((f"c4 {tag} N={n} K={k}",
                               [(f"c4 {tag} {m}x{n}x{k}", m, n, k, (edt, tdt), "uniform", None) for m in (128, 512, 2048)]))
    dev = f"cuda:{device}"
    out, group_clocks = [], []
    torch.backends.cuda.matmul.allow_tf32 = False  # the cuBLAS comparison of fp32 data is a true fp32 GEMM
    for gname, cases in groups:
        t_g0 = time.time()
        for tag, m, n, k, (edt, tdt), dist, keys in cases:
            try:
                kpm = tuned_config(m, n, k, edt) if keys is None else default_config(m, n, k, edt, **keys)
                inc, kern = build_kernel(kpm, device)
                A, B = seeded_operands(m, n, k, tdt, dist, seed=0)
                eb = A.element_size()
                nbytes = eb * (m * k + k * n + m * n)
                copies = 1 if nbytes > L2_BYTES else int(2 * L2_BYTES // nbytes) + 2
                sets = [(A.to(dev), B.to(dev), torch.empty(m, n, dtype=tdt, device=dev)) for _ in range(copies)]
                del A, B
                turn = [0]

                def ours():
                    a, b, c = sets[turn[0] % copies]
                    turn[0] += 1
                    kern.run(a, b, c)

                def cublas():
                    a, b, c = sets[turn[0] % copies]
                    turn[0] += 1
                    torch.matmul(a, b, out=c)

                ts = sorted(time_launches(ours, launches, 3))
                kern.checkStatus()
                g_ours = time_graph(ours, launches)
                kern.checkStatus()
                a0, b0, c0 = sets[0]
                kern.run(a0, b0, c0)
                mine = c0.clone()
                tl = sorted(time_launches(cublas, launches, 3))
                g_lib = time_graph(cublas, launches)
                torch.matmul(a0, b0, out=c0)
                scale = c0.float().abs().max().clamp_min(1e-30)
                diff = float(((mine.float() - c0.float()).abs().max() / scale).item())
                med, lib_med = ts[len(ts) // 2], tl[len(tl) // 2]
                flops = rl.gemm_flops(m, n, k)
                variant = int(inc.kernelInfo["kernel"])
                parts = variant == KERNEL_F32_SPLIT  # three fp16 products a step
                tensor_peak = (rl.tensor_peak_tflops("bfloat16", False, peaks) / 3 if parts else
                               rl.tensor_peak_tflops(str(tdt).replace("torch.", ""), variant == 1, peaks))
                roof = rl.shape_roofline(m, n, k, eb, tensor_peak, peaks["hbm_gbs"])
                bound, peak = roof["bound"], roof["peak"]
                tfl = flops / (med * 1e9)
                out.append({
                    "workload": tag, "dtype": "f32(fp16 parts)" if parts else "f32(3xtf32)" if (tdt == torch.float32 and variant != 1) else
                    ("f32" if tdt == torch.float32 else "bf16"), "ms": round(med, 4), "ms_best": round(ts[0], 4),
                    "tflops": round(tfl, 1), "gbs": round(nbytes / med / 1e6, 0),
                    "roofline": {"bound": bound, "peak": round(peak, 1), "frac": round(tfl / peak, 4),
                                 "peak_source": ("FFMA pipe 74 TFLOP/s" if variant == 1 else
                                                 f"{peaks['source']} bf16_tflops / 3" if parts else
                                                 "nominal TF32 1100 / 3" if tdt == torch.float32 else
                                                 f"{peaks['source']} bf16_tflops") +
                                                (f", capped by AI x {peaks['source']} hbm_gbs" if bound == "hbm" else "")},
                    "cublas_tflops": round(flops / (lib_med * 1e9), 1), "vs_cublas": round(lib_med / med, 3),
                    "graph_replay": None if (g_ours is None or g_lib is None) else {
                        "ms": round(g_ours, 4), "tflops": round(flops / (g_ours * 1e9), 1),
                        "cublas_ms": round(g_lib, 4), "vs_cublas": round(g_lib / g_ours, 3)},
                    "max_diff_vs_cublas_rel": diff,
                    "tile": f"{kpm.BLOCK_SIZE_M}x{kpm.BLOCK_SIZE_N}x{kpm.BLOCK_SIZE_K}", "split_k": int(kpm.LOCAL_SPLIT_U),
                    "kernel_variant": variant, "launches": launches,
                    "l2": "larger than L2" if copies == 1 else f"cold: rotates over {copies} operand sets",
                    "group": gname})
                del sets, mine, a0, b0, c0
                torch.cuda.empty_cache()
            except Exception as e:  # a secondary figure must not lose the headline line
                out.append({"workload": tag, "group": gname, "error": str(e)[:300]})
        group_clocks.append(dict(sampler.window(t_g0, time.time(), gname), group=gname))
    return out, group_clocks


def chain_workloads(device: int, sampler: "ClockSampler", launches: int = 20):
    """The operators around the plain product (batched, strided, attention-shaped chain), each timed like the
    workloads above beside the PyTorch library call for the same thing and checked against the host composition
    at fp32 (the oracle's ``torch.matmul`` plus ``torch.softmax``): a sample of the result, outside the timing."""
    import torch
    from oracle import oracle
    from codegendemo_b200.kcg import matmul_op
    dev = f"cuda:{device}"
    out = []
    t_g0 = time.time()
    g = torch.Generator().manual_seed(0)

    def entry(tag, flops, ours, lib, lib_name, max_rel, note):
        ts = sorted(time_launches(ours, launches, 3))
        tl = sorted(time_launches(lib, launches, 3))
        g_ours, g_lib = time_graph(ours, launches), time_graph(lib, launches)
        med, lib_med = ts[len(ts) // 2], tl[len(tl) // 2]
        out.append({"workload": tag, "dtype": "bf16", "ms": round(med, 4), "ms_best": round(ts[0], 4),
                    "tflops": round(flops / (med * 1e9), 1), "library": lib_name,
                    "library_tflops": round(flops / (lib_med * 1e9), 1), "vs_library": round(lib_med / med, 3),
                    "graph_replay": None if (g_ours is None or g_lib is None) else {
                        "ms": round(g_ours, 4), "library_ms": round(g_lib, 4), "vs_library": round(g_lib / g_ours, 3)},
                    "oracle_check": {"max_rel": max_rel, "tol": TOL_16BIT, "ok": bool(max_rel <= TOL_16BIT),
                                     "against": note}, "launches": launches, "group": "operators around the product"})

    def rel(got, ref):
        ref = ref.float()
        return float(((got.float().cpu() - ref).abs().max() / ref.abs().max().clamp_min(1e-30)).item())

    try:  # batched product: 16 x (1024 x 1024 x 1024)
        a = (torch.randn(16, 1024, 1024, generator=g) / 32).bfloat16().to(dev)
        b = (torch.randn(16, 1024, 1024, generator=g) / 32).bfloat16().to(dev)
        c = torch.empty(16, 1024, 1024, dtype=torch.bfloat16, device=dev)
        matmul_op.bmm(a, b, c)
        err = max(rel(c[i], oracle.host_matmul(a[i], b[i])) for i in (0, 15))
        entry("bmm bf16 16 x 1024^3", 2.0 * 16 * 1024 ** 3, lambda: matmul_op.bmm(a, b, c),
              lambda: torch.bmm(a, b, out=c), "torch.bmm (cuBLAS)", err, "host torch.matmul fp32 of batches 0 and 15")
        del a, b, c
    except Exception as e:
        out.append({"workload": "bmm bf16 16 x 1024^3", "error": str(e)[:300]})
    try:  # operands with a row pitch: column blocks of wider tensors, nothing copied
        wide_a = (torch.randn(2048, 8192, generator=g) / 64).bfloat16().to(dev)
        wide_b = (torch.randn(4096, 8192, generator=g) / 64).bfloat16().to(dev)
        wide_c = torch.zeros(2048, 8192, dtype=torch.bfloat16, device=dev)
        av, bv, cv = wide_a[:, 4096:], wide_b[:, :4096], wide_c[:, 2048:6144]
        matmul_op.matmul(av, bv, c=cv)
        rows = slice(512, 640)
        err = rel(cv[rows], oracle.host_matmul(av[rows], bv))
        untouched = bool((wide_c[:, :2048] == 0).all().item() and (wide_c[:, 6144:] == 0).all().item())
        entry("strided bf16 2048x4096x4096 (column blocks of 8192-wide tensors)", 2.0 * 2048 * 4096 * 4096,
              lambda: matmul_op.matmul(av, bv, c=cv), lambda: torch.matmul(av, bv, out=cv), "torch.matmul on the views",
              err if untouched else float("inf"), "host torch.matmul fp32 of rows 512..639; C outside the block stays zero")
        del wide_a, wide_b, wide_c
    except Exception as e:
        out.append({"workload": "strided bf16 2048x4096x4096", "error": str(e)[:300]})
    try:  # attention-shaped chain: 16 heads x 2048 x 128
        H, S, D = 16, 2048, 128
        q, k, v = ((torch.randn(H, S, D, generator=g)).bfloat16().to(dev) for _ in range(3))
        o = matmul_op.attention(q, k, v)
        ref = torch.softmax(oracle.host_matmul(q[3], k[3].t().contiguous()) / math.sqrt(D), dim=-1) @ v[3].float().cpu()
        err = rel(o[3], ref)
        entry(f"attention chain bf16 {H} heads x {S} x {D}", 4.0 * H * S * S * D, lambda: matmul_op.attention(q, k, v, out=o),
              lambda: torch.nn.functional.scaled_dot_product_attention(q[None], k[None], v[None]),
              "torch scaled_dot_product_attention (fused library kernel, scores never materialised)", err,
              "host softmax(q k^T / sqrt(d)) v at fp32, head 3")
        o2 = matmul_op.attention_fused(q, k, v)
        matmul_op.attention_status(device)
        entry(f"attention fused kernel bf16 {H} heads x {S} x {D}", 4.0 * H * S * S * D,
              lambda: matmul_op.attention_fused(q, k, v, out=o2),
              lambda: torch.nn.functional.scaled_dot_product_attention(q[None], k[None], v[None]),
              "torch scaled_dot_product_attention (fused library kernel)", rel(o2[3], ref),
              "host softmax(q k^T / sqrt(d)) v at fp32, head 3")
        matmul_op.attention_status(device)
        del q, k, v, o, o2
        H, S, D = 32, 8192, 128  # a longer sequence, fused kernel only (the chain would materialise 8 GB of scores)
        q, k, v = ((torch.randn(H, S, D, generator=g)).bfloat16().to(dev) for _ in range(3))
        o2 = matmul_op.attention_fused(q, k, v)
        ref = torch.softmax(oracle.host_matmul(q[7, :256], k[7].t().contiguous()) / math.sqrt(D), dim=-1) @ v[7].float().cpu()
        entry(f"attention fused kernel bf16 {H} heads x {S} x {D}", 4.0 * H * S * S * D,
              lambda: matmul_op.attention_fused(q, k, v, out=o2),
              lambda: torch.nn.functional.scaled_dot_product_attention(q[None], k[None], v[None]),
              "torch scaled_dot_product_attention (fused library kernel)", rel(o2[7, :256], ref),
              "host softmax(q k^T / sqrt(d)) v at fp32, head 7, rows 0..255")
        matmul_op.attention_status(device)
        del q, k, v, o2
    except Exception as e:
        out.append({"workload": "attention bf16", "error": str(e)[:300]})
    torch.cuda.empty_cache()
    return out, dict(sampler.window(t_g0, time.time(), "operators around the product"), group="operators around the product")


# ------------------------------------------------------------------------------------ CPU legs
class CpuGemm:
    """The reference's CPU path for this workload: ``torch.matmul`` on host tensors, bf16 operands up-cast to
    fp32 (as the oracle computes), all host threads. Operands are built ONCE here; `timed_pass` holds nothing
    but the call between its two timestamps."""

    def __init__(self, A_bf16, B_bf16, threads: int, budget_s: float, passes: int):
        import torch
        torch.set_num_threads(threads)
        self.threads = threads
        Bf = B_bf16.float()
        probe = A_bf16[:256].float()
        torch.matmul(probe, Bf)  # warm the BLAS threads
        t0 = time.perf_counter()
        torch.matmul(probe, Bf)
        per_row = (time.perf_counter() - t0) / 256
        # all rows if `passes` passes of them fit the budget, else the largest 128-row multiple that does
        rows = A_bf16.shape[0]
        if per_row * rows * passes > budget_s:
            rows = max(1024, int(budget_s / passes / per_row) // 128 * 128)
        self.rows = min(rows, A_bf16.shape[0])
        self.Af, self.Bf = A_bf16[:self.rows].float(), Bf
        self.flops = 2.0 * self.rows * Bf.shape[1] * Bf.shape[0]

    def timed_pass(self) -> float:
        import torch
        t0 = time.perf_counter()
        torch.matmul(self.Af, self.Bf)
        return time.perf_counter() - t0

    def sample(self) -> str:
        what = "the whole product" if self.rows == M_TOTAL else f"a {self.rows}-row slab of A"
        return (f"{what} ({self.rows}x{K_SIZE} times {K_SIZE}x{N_SIZE}) per pass, torch.matmul fp32 on host tensors "
                f"(the reference's oracle call), operands resident before the clock starts")


def workload_config(n_gpus):
    return {"workload": f"bf16 NN GEMM M=32768 N=8192 K=8192 sharded by M over {n_gpus} GPU(s), B replicated, "
                        "C sharded (at 1 GPU the whole product); inputs normal(0,1)/sqrt(K), CPU generator seed 0",
            "m": M_TOTAL, "n": N_SIZE, "k": K_SIZE, "rows_per_gpu": M_TOTAL // n_gpus,
            "l2": "inputs larger than L2 (A slab + B + C slab >= 256 MiB per GPU); no flush"}


def run_reference(args, rank, world):
    if rank != 0:
        return 0
    import torch
    threads = os.cpu_count() or 1
    A, B = seeded_operands(M_TOTAL, N_SIZE, K_SIZE, torch.bfloat16, "normal", seed=0)
    cpu = CpuGemm(A, B, threads, budget_s=120.0, passes=max(1, args.steps + args.warmup))
    del A, B
    for _ in range(args.warmup):
        cpu.timed_pass()
    total = 0.0
    for _ in range(args.steps):
        total += cpu.timed_pass()
    dt = total / max(1, args.steps)
    val = cpu.flops / dt / 1e12
    line = {
        "impl": "reference", "metric": METRIC, "value": round(val, 4), "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(dt * 1e3, 3), "higher_is_better": True,
        "scaling": "strong", "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
        "config": workload_config(args.gpus),
        "cpu_baseline": {"value": round(val, 4), "unit": UNIT, "cores": threads, "kind": "port", "sample": cpu.sample()},
        "e2e": {"value": round(val, 4), "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--e2e-steps", type=int, default=20)
    ap.add_argument("--no-extras", action="store_true", help="skip other_workloads and cpu_baseline")
    ap.add_argument("--extras-only-operators", action="store_true",
                    help="of other_workloads run only the operators around the product (batched, strided, attention)")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3) if args.impl == "ours" else args.warmup
    rank, local_rank, world = env_int("RANK", 0), env_int("LOCAL_RANK", 0), env_int("WORLD_SIZE", 1)

    if args.impl == "reference":
        return run_reference(args, rank, world)

    import torch
    import torch.distributed as dist
    from codegendemo_b200 import _lib
    from codegendemo_b200.kcg import dist as kdist

    if not torch.cuda.is_available():
        raise SystemExit("bench.py needs a CUDA device: the GEMM path has no CPU fallback")
    if world > 1:
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        dist.init_process_group("nccl", device_id=torch.device(f"cuda:{local_rank}"))
    torch.cuda.set_device(local_rank)
    dev = f"cuda:{local_rank}"
    n_gpus = world
    row0, row1 = kdist.shard_rows(M_TOTAL, n_gpus, rank, 256)
    rows = row1 - row0

    # Seeded synthetic operands (see seeded_operands): every rank draws the same A and B and keeps its row slab.
    A_full, B_host = seeded_operands(M_TOTAL, N_SIZE, K_SIZE, torch.bfloat16, "normal", seed=0)
    A_host = A_full[row0:row1].contiguous()
    if n_gpus > 1:
        del A_full
    a = A_host.to(dev)
    b = B_host.to(dev)
    kdist.replicate_b(b, src=0)  # every rank holds the same B before timing (the bytes already agree)
    c = torch.full((rows, N_SIZE), float("nan"), dtype=torch.bfloat16, device=dev)

    kpm, (inc, kern) = build_bf16_kernel(rows, local_rank)
    kernel_desc = (f"tile {kpm.BLOCK_SIZE_M}x{kpm.BLOCK_SIZE_N}x{kpm.BLOCK_SIZE_K}, {inc.kernelInfo['stages']} stages, "
                   + ("tcgen05 cta_group::2 on CTA pairs" if inc.kernelInfo["kernel"] == 4 else "tcgen05 cta_group::1")
                   + f", persistent grid {inc.m_gridDims[0]}")
    lib = _lib.get_lib()
    kern.run(a, b, c)  # first launch loads the module
    kern.checkStatus()

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()
        time.sleep(0.3)
    barrier()
    t_loaded0 = time.time()
    for _ in range(args.warmup):
        kern.run(a, b, c)
    launches0 = lib.kcg_launch_count()
    barrier()
    t_timed0 = time.time()
    evs = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps + 1)]
    evs[0].record()
    for i in range(args.steps):
        kern.run(a, b, c)
        evs[i + 1].record()
    barrier()
    t_timed1 = time.time()
    launches = lib.kcg_launch_count() - launches0
    total_ms = evs[0].elapsed_time(evs[-1])
    per_launch = [evs[i].elapsed_time(evs[i + 1]) for i in range(args.steps)]
    # nvidia-smi needs tens of ms per sample; a short timed region may hold none. The same launches
    # are then continued, untimed, for ~0.4 s on every rank so that the clocks are sampled under this
    # very load (the window label in `clocks` says which samples were used).
    t_cont0 = time.time()
    if (t_timed1 - t_loaded0) < 0.35:
        n_more = max(1, int(0.4 / max(total_ms / args.steps / 1e3, 1e-5)))
        for _ in range(n_more):
            kern.run(a, b, c)
        barrier()
    t_cont1 = time.time()
    clocks = None
    if rank == 0:
        used = sampler.window(t_timed0, t_timed1, "timed region")
        if used["samples"] < 3:
            used = sampler.window(t_loaded0, t_cont1, "warm-up + timed region" + (
                " + untimed continuation of the same launches" if t_cont1 - t_cont0 > 0.05 else ""))
        clocks = used
    kern.checkStatus()
    total_ms = kdist.max_over_ranks(total_ms, device=dev)
    ms_per_step = total_ms / args.steps
    flops_total = 2.0 * M_TOTAL * N_SIZE * K_SIZE
    value = flops_total / (ms_per_step * 1e9)

    # ---- parity, outside the timed region: this rank's slab against the CPU oracle
    check = oracle_check(c, A_host, B_host, full=(n_gpus == 1), blocks=8, seed=rank)
    check["max_rel"] = kdist.max_over_ranks(check["max_rel"], device=dev)
    check["ok"] = kdist.max_over_ranks(0.0 if check["ok"] else 1.0, device=dev) == 0.0
    check["ranks_checked"] = n_gpus

    # roofline of the one kernel in the step (this rank's launches)
    peaks = measured_peaks()
    avg_launch_ms = sum(per_launch) / len(per_launch)
    achieved = 2.0 * rows * N_SIZE * K_SIZE / (avg_launch_ms * 1e9)
    timed_s = total_ms / 1e3
    # the power cap pulls the clock down after roughly 0.1 s of dense MMA: longer regions are scored
    # against the sustained cuBLAS figure, shorter ones against the burst figure
    peak_kind = "bf16_tflops_sustained" if timed_s > 0.1 else "bf16_tflops"
    peak = peaks[peak_kind]
    # DRAM traffic of one launch (dram__bytes_read.sum + dram__bytes_write.sum, one-pass ncu captures, see
    # profiles/): 512x256 pair tile 5.76 GB for the full 32768-row launch and 1.95 GB for a 16384-row launch (the
    # re-reads grow faster than the rows: more raster groups stream B through L2); 275.0 MB for a 2048-row launch
    # of the 256x256x128 pair tile (the tile of the 4096-row slabs); 227.4 MB for a 2048-row launch of the
    # single-CTA kernel. Other slab heights are scaled by their rows from the nearest measured one.
    if inc.kernelInfo["kernel"] == 4 and kpm.BLOCK_SIZE_M == 512:
        traffic = 5.76e9 * rows / 32768.0 if rows > 16384 else 1.95e9 * rows / 16384.0
    elif inc.kernelInfo["kernel"] == 4:
        traffic = 275.0e6 * rows / 2048.0
    else:
        traffic = 227.4e6 * rows / 2048.0
    roofline = {"bound": "tensor", "achieved": round(achieved, 1), "peak": peak, "unit": "TFLOP/s",
                "frac": round(achieved / peak, 4), "traffic": traffic,
                "peak_source": f"{peaks['source']} {peak_kind} (cuBLAS bf16 8192^3)",
                "frac_of_nominal_2250": round(achieved / 2250.0, 4), "kernel_ms": round(avg_launch_ms, 4)}

    # end to end through the C ABI with host buffers: H2D(A slab, B) + kernel + D2H(C slab) per step
    hA = A_host.pin_memory()
    hB = B_host.pin_memory()
    hC = torch.empty(rows, N_SIZE, dtype=torch.bfloat16).pin_memory()
    kern.runHost(hA, hB, hC)  # warm-up (allocates the library's device buffers)
    barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(args.e2e_steps):
        kern.runHost(hA, hB, hC)
    e1.record()
    barrier()
    own_e2e_ms = e0.elapsed_time(e1) / args.e2e_steps
    e2e_ms = kdist.max_over_ranks(own_e2e_ms, device=dev)
    h2d_rank, d2h_rank = int(hA.numel() * 2 + hB.numel() * 2), int(hC.numel() * 2)
    e2e = {"value": round(flops_total / (e2e_ms * 1e9), 2), "unit": UNIT, "ms_per_step": round(e2e_ms, 3),
           "h2d_bytes_per_step": h2d_rank * n_gpus, "d2h_bytes_per_step": d2h_rank * n_gpus, "steps": args.e2e_steps,
           # copies in both directions overlap inside a step, so each rate is that direction's bytes over the whole step
           "per_rank": {"h2d_bytes": h2d_rank, "d2h_bytes": d2h_rank,
                        "h2d_gbs": round(h2d_rank / e2e_ms / 1e6, 1), "d2h_gbs": round(d2h_rank / e2e_ms / 1e6, 1),
                        "note": "every rank re-sends the replicated B each step; all ranks share one host"},
           "api": "kcg_matmul_host (CompiledKernel.runHost), pinned host buffers"}
    # The host entry runs row slabs, whose last-wave K split can differ from the whole-slab launch:
    # equal up to fp32 summation order, i.e. a rare last-bit difference after rounding to bf16.
    dev_c = c.cpu().float()
    e2e_diff = float(((hC.float() - dev_c).abs().max() / dev_c.abs().max().clamp_min(1e-30)).item())
    same = bool(e2e_diff <= 1e-2)
    # and the host-buffer result against the oracle too (same sampled blocks)
    e2e_check = oracle_check(hC, A_host, B_host, full=False, blocks=8, seed=rank)
    e2e["oracle_check"] = {"blocks": e2e_check["blocks"],
                           "max_rel": kdist.max_over_ranks(e2e_check["max_rel"], device=dev),
                           "tol": TOL_16BIT,
                           "ok": kdist.max_over_ranks(0.0 if e2e_check["ok"] else 1.0, device=dev) == 0.0}

    # Optional collective, timed apart from the GEMM: all-gather of the C slabs (NCCL over NVLink).
    allgather = None
    if world > 1:
        c_full = torch.empty(M_TOTAL, N_SIZE, dtype=torch.bfloat16, device=dev)
        for _ in range(2):
            kdist.all_gather_c(c, c_full)
        barrier()
        g0, g1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        n_ag = 5
        g0.record()
        for _ in range(n_ag):
            kdist.all_gather_c(c, c_full)
        g1.record()
        barrier()
        ag_ms = kdist.max_over_ranks(g0.elapsed_time(g1) / n_ag, device=dev)
        recv = (n_gpus - 1) * rows * N_SIZE * 2  # bytes each rank receives
        allgather = {"ms": round(ag_ms, 4), "recv_bytes_per_rank": recv,
                     "recv_gbs_per_rank": round(recv / ag_ms / 1e6, 1),
                     "bus_gbs": round(recv / ag_ms / 1e6, 1),  # all-gather bus bandwidth = (n-1)/n * total / t
                     "correct": bool(torch.equal(c_full[row0:row1], c)), "note": "not part of value / ms_per_step"}
        # The same product with the all-gather fused into the kernel: every finished tile is stored
        # into the full C of all GPUs (peer buffers mapped through CUDA IPC, stores over NVLink).
        # Nothing waits inside the kernel; a step is complete when every rank's launch has completed.
        sym = kdist.SymmetricC(M_TOTAL, N_SIZE, 2, rank, world, local_rank)
        full = sym.full(torch.bfloat16)
        full.zero_()
        barrier()
        # Two tiles are tried: the GEMM's own, and 128x256 whose two TMEM accumulator buffers let the
        # epilogue overlap the next tile's main loop.
        from codegendemo_b200.kcg.matmul_op import build_kernel, default_config
        from codegendemo_b200.kcg.Utils import EnumKernelDType as E
        _, kern_ov = build_kernel(default_config(rows, N_SIZE, K_SIZE, E.bfloat16), local_rank)
        n_f = 10
        fused_by_tile, fused_ok = {}, {}
        for label, kf in (("gemm_tile", kern), ("128x256x64", kern_ov)):
            full.zero_()
            barrier()  # every copy is cleared before any rank stores into it
            for _ in range(3):
                kdist.matmul_allgather(kf, a, b, sym)
            barrier()
            f0, f1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            f0.record()
            for _ in range(n_f):
                kdist.matmul_allgather(kf, a, b, sym)
            f1.record()
            barrier()
            fused_by_tile[label] = round(kdist.max_over_ranks(f0.elapsed_time(f1) / n_f, device=dev), 4)
            kf.checkStatus()
            barrier()
            # every rank checks the FULL matrix it holds against the NCCL-gathered one. Another tile may
            # K-split its last wave differently: equal up to fp32 summation order (a last-bit difference
            # after rounding to bf16), bit for bit with the GEMM's own tile.
            diff = float(((full.float() - c_full.float()).abs().max() / c_full.float().abs().max()).item())
            ok_here = bool(torch.equal(full, c_full)) if label == "gemm_tile" else diff <= 1e-2
            fused_ok[label] = kdist.max_over_ranks(0.0 if ok_here else 1.0, device=dev) == 0.0
            barrier()
        # ... and against the CPU oracle: a 128-row block of ANOTHER rank's rows, as this GPU received it
        other = (rank + 1) % world
        A_all, _ = seeded_operands(M_TOTAL, N_SIZE, K_SIZE, torch.bfloat16, "normal", seed=0)
        r_chk = other * rows + 128 * (rank % max(1, rows // 128))
        from oracle import oracle
        ref_blk = oracle.host_matmul(A_all[r_chk:r_chk + 128], B_host)
        del A_all
        g_err, g_nan = rel_error(full[r_chk:r_chk + 128].cpu().float(), ref_blk)
        gathered_ok = kdist.max_over_ranks(0.0 if (g_err <= TOL_16BIT and not g_nan) else 1.0, device=dev) == 0.0
        fused_ms = min(fused_by_tile.values())
        sent = (n_gpus - 1) * rows * N_SIZE * 2
        allgather["fused_into_gemm"] = {
            "ms": round(fused_ms, 4), "ms_by_tile": fused_by_tile,
            "gemm_then_nccl_allgather_ms": round(ms_per_step + ag_ms, 4),
            "tflops": round(flops_total / (fused_ms * 1e9), 1), "sent_bytes_per_rank": sent,
            "nvlink_gbs_per_rank": round(sent / fused_ms / 1e6, 1),
            "nvlink_floor_ms_at_770_gbs": round(sent / 770e9 * 1e3, 4),
            "correct": all(fused_ok.values()), "correct_by_tile": fused_ok,
            "oracle_check_of_received_rows": {"max_rel": kdist.max_over_ranks(g_err, device=dev), "tol": TOL_16BIT,
                                              "ok": gathered_ok},
            "api": "kcg_launch_gemm_allgather (kcg.dist.matmul_allgather)"}
        barrier()
        sym.close()
        barrier()
        sym.free()
        del c_full, full

    extras, group_clocks, cpu_base = None, None, None
    if rank == 0 and n_gpus == 1 and not args.no_extras:
        del hA, hB, hC
        extras, group_clocks = ([], []) if args.extras_only_operators else other_workloads(local_rank, peaks, sampler)
        chain, chain_clocks = chain_workloads(local_rank, sampler)
        extras += chain
        group_clocks.append(chain_clocks)
        threads = os.cpu_count() or 1
        cpu = CpuGemm(A_full, B_host, threads, budget_s=20.0, passes=4)
        secs = [cpu.timed_pass() for _ in range(4)]
        best = min(secs)
        cpu_base = {"value": round(cpu.flops / best / 1e12, 4), "unit": UNIT, "cores": threads, "kind": "port",
                    "sample": cpu.sample() + f"; best of {len(secs)} passes of {best:.2f} s"}
    if rank == 0:
        sampler.stop()
        line = {
            "metric": METRIC, "value": round(value, 1), "unit": UNIT, "n_gpus": n_gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": round(ms_per_step, 4), "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
            "config": workload_config(n_gpus), "kernel": kernel_desc, "roofline": roofline,
            "oracle_check": check, "cpu_baseline": cpu_base, "e2e": e2e,
            "gpu_launches": int(launches), "clocks": clocks, "e2e_matches_device_result": same,
            "e2e_max_diff_vs_device_rel": e2e_diff,
            "allgather_c": allgather,
        }
        if extras is not None:
            sys.stderr.write(json.dumps({"other_workloads": extras, "other_workloads_clocks": group_clocks}) + "\n")
            sys.stderr.flush()
        print(json.dumps(line), flush=True)
    ok = check["ok"] and e2e["oracle_check"]["ok"]
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    if not ok:
        sys.stderr.write(f"oracle check FAILED: {check} / e2e {e2e['oracle_check']}\n")
        return 1
    return 0


if __name__ == "__main__":
    sys.exit(main())
