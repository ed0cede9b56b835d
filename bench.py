#!/usr/bin/env python
"""Benchmark of the Strata transformer-block hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]

Workload (the reference benchmark's single-GPU configuration): one bf16 Strata backbone block forward over a batch of
4 tiles of 16 x 64 x 64 tokens, dim 512, 8 heads x 64, 3-D neighbourhood kernel (3,9,9),
stereographic RoPE, MLP ratio 4 tanh-GELU; N(0,1) activations, trunc-normal(0.02) weights,
all synthetic. A "step" is one block forward over the batch. With N > 1 GPUs every rank
runs its own batch of 4 tiles (tiles are the sharding unit; weak scaling).

Prints ONE JSON line: metric "block_tokens_per_s" (whole job), the roofline of the dominant
kernel, a CPU baseline (the fp32 oracle restatement timed on the host cores), the end-to-end
number through the C ABI with host buffers, clocks sampled during the timed region. The same
line carries the strong-scaling steps that contain the halo exchange ("step": 12 blocks over 24
tiles, K/V halo in every block; "global_step": 24 blocks of dim 1024 over 96 tiles with a
16-token halo, run as a rollout), whose times shrink with N where the headline's does not.
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

WORKLOAD = dict(workload="strata_block_fwd_bf16", tiles_per_gpu=4, token_grid=[16, 64, 64],
                dim=512, heads=8, head_dim=64, kernel=[3, 9, 9], mlp_ratio=4, rope="stereographic",
                gated=False, qk_norm=False, l2="inputs_exceed_l2 (2.9 GB touched per step)")
CPU_SAMPLE = dict(tiles=2, token_grid=[8, 32, 32])   # bounded sample of the same workload


def flops_per_token(C, kernel, ratio=4.0):
    K = kernel[0] * kernel[1] * kernel[2]
    return 6 * C * C + 4 * K * C + 2 * C * C + 4 * ratio * C * C


# DRAM bytes per launch (dram__bytes_read.sum + dram__bytes_write.sum) from the ncu captures
# summarised under profiles/ (same workload, one launch each).
NCU_TRAFFIC_BYTES = {"na3d_fwd": 1.199e9, "gemm_fc1_gelu": 1.288e9, "gemm_qkv_rope": 1.022e9}


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["bf16_tflops"]), float(d["hbm_gbs"]), "measured"
    return 1590.0, 6650.0, "fallback"


def sustained_tflops():
    """cuBLAS bf16 throughput in a seconds-long loop under the power cap (the denominator for a
    step timed inside a long region)."""
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        return float(json.loads(p.read_text()).get("bf16_tflops_sustained", 1400.0))
    return 1400.0


# --------------------------------------------------------------------------- CPU reference arm
def cpu_block_tokens_per_s(steps: int, warmup: int, threads: int | None = None):
    """Times the fp32 oracle block (CPU restatement of the reference block; physicsnemo and
    NATTEN are not installable here) on a bounded sample of the workload."""
    import torch
    from oracle import block_oracle as bo
    threads = threads or os.cpu_count() or 1
    torch.set_num_threads(threads)
    C, heads, kernel = WORKLOAD["dim"], WORKLOAD["heads"], tuple(WORKLOAD["kernel"])
    D, H, W = CPU_SAMPLE["token_grid"]
    n = CPU_SAMPLE["tiles"]
    p = bo.init_block_params(C, seed=0)
    g = torch.Generator().manual_seed(0)
    x = torch.randn(n, D * H * W, C, generator=g)
    lat = torch.linspace(0.2, 0.7, H).view(1, H, 1).expand(n, H, W)
    lon = torch.linspace(0.1, 0.6, W).view(1, 1, W).expand(n, H, W)
    cos, sin = bo.stereographic_rope_tables(lat, lon, C // heads, 1, bo.default_rope_length_scale(1))
    run = lambda: bo.block_forward(x, p, grid=(D, H, W), num_heads=heads, kernel=kernel,
                                   rope_cos=cos, rope_sin=sin)
    with torch.no_grad():
        for _ in range(warmup):
            run()
        t0 = time.perf_counter()
        for _ in range(steps):
            run()
        dt = (time.perf_counter() - t0) / steps
    tokens = n * D * H * W
    return tokens / dt, dt * 1e3, threads, f"{n} tile of {D}x{H}x{W} tokens, dim {C}, kernel {list(kernel)}, fp32"


def cpu_config1_block_ms(threads: int = 8, runs: int = 5):
    """The reference benchmark's CPU configuration: one tile of 8 x 32 x 32 tokens, dim 128,
    4 heads x 32, kernel (3, 7, 7), stereographic RoPE, MLP ratio 4, Xavier weights, fp32, on
    8 host threads; median of `runs` after a warm-up. (Timed with the oracle restatement of the
    block: physicsnemo / NATTEN are not installable here.)"""
    import torch
    from oracle import block_oracle as bo
    prev = torch.get_num_threads()
    torch.set_num_threads(min(threads, os.cpu_count() or 1))
    try:
        C, heads, kernel, (D, H, W) = 128, 4, (3, 7, 7), (8, 32, 32)
        p = bo.init_block_params(C, seed=0, scheme="xavier")
        x = torch.randn(1, D * H * W, C, generator=torch.Generator().manual_seed(0))
        lat = torch.linspace(0.2, 0.7, H).view(1, H, 1).expand(1, H, W)
        lon = torch.linspace(0.1, 0.6, W).view(1, 1, W).expand(1, H, W)
        cos, sin = bo.stereographic_rope_tables(lat, lon, C // heads, 1, bo.default_rope_length_scale(1))
        run = lambda: bo.block_forward(x, p, grid=(D, H, W), num_heads=heads, kernel=kernel,
                                       rope_cos=cos, rope_sin=sin)
        ts = []
        with torch.no_grad():
            run()
            for _ in range(runs):
                t0 = time.perf_counter()
                run()
                ts.append((time.perf_counter() - t0) * 1e3)
        ms = statistics.median(ts)
        return {"ms": ms, "tokens_per_s": D * H * W / (ms * 1e-3), "cores": torch.get_num_threads(),
                "kind": "port", "workload": "1 tile 8x32x32 tokens, dim 128, 4x32 heads, kernel [3,7,7], fp32"}
    finally:
        torch.set_num_threads(prev)


def cpu_face_halo_ms(n: int = 1024, pad: int = 32, channels: int = 8, runs: int = 3):
    """CPU time of the face-level copy / rot90 / corner halo (the reference's
    create_padded_faces_batched, screamcast/cubesphere_transforms.py:357-445, here its numpy
    restatement) on `channels` x 6 faces of n x n cells with a halo of `pad`."""
    import numpy as np
    from oracle import halo_oracle as ho
    x = np.random.default_rng(0).standard_normal((channels, 6, n, n)).astype(np.float32)
    ho.create_padded_faces(x, pad)
    ts = []
    for _ in range(runs):
        t0 = time.perf_counter()
        ho.create_padded_faces(x, pad)
        ts.append((time.perf_counter() - t0) * 1e3)
    ms = statistics.median(ts)
    return {"ms": ms, "gbs": (x.nbytes + x.nbytes * ((n + 2 * pad) / n) ** 2) / (ms * 1e-3) / 1e9,
            "cores": 1, "kind": "port", "workload": f"{channels} x 6 faces of {n}x{n} fp32, halo {pad}"}


def run_reference_arm(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    steps = max(1, min(args.steps, 3))
    warm = 1
    tps, ms, threads, sample = cpu_block_tokens_per_s(steps, warm)
    line = {
        "impl": "reference", "metric": "block_tokens_per_s", "value": tps, "unit": "tokens/s",
        "n_gpus": args.gpus, "steps": steps, "warmup": warm, "ms_per_step": ms,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
        "data": "synthetic", "config": dict(WORKLOAD, sample=sample),
        "cpu_baseline": {"value": tps, "unit": "tokens/s", "cores": threads, "kind": "port",
                         "sample": sample},
        "cpu_baseline_config1": cpu_config1_block_ms(),
        "e2e": {"value": tps, "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "note": "CPU restatement of the reference block (physicsnemo / NATTEN unavailable here)",
    }
    print(json.dumps(line), flush=True)


# --------------------------------------------------------------------------- clocks
class ClockSampler:
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.tmp = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu}", f"--query-gpu={self.Q}",
                 "--format=csv,noheader,nounits", "-lms", "20"],
                stdout=self.tmp, stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self):
        out = {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}
        if self.proc is None:
            return out
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.tmp.flush()
        rows = [r.split(", ") for r in Path(self.tmp.name).read_text().strip().splitlines() if r]
        os.unlink(self.tmp.name)
        sm, reasons = [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in rows:
            if len(r) < 9:
                continue
            try:
                sm.append(float(r[1]))
                out["sm_max_mhz"] = float(r[2])
            except ValueError:
                continue
            for nm, val in zip(names, r[5:9]):
                if val.strip().lower().startswith("active"):
                    reasons.add(nm)
        if sm:
            # median over the busiest half of the samples (the sampler also sees idle time)
            sm.sort()
            out["sm_mhz"] = statistics.median(sm)
            out["samples"] = len(sm)
        out["reasons"] = sorted(reasons)
        return out


# --------------------------------------------------------------------------- GPU arm
def bind_to_gpu_cpus(gpu_index: int):
    """Multi-rank runs: restrict this rank to the CPUs NVML reports as local to its GPU, so that
    the pinned host buffers of the end-to-end leg are first-touched on the GPU's own NUMA node
    (eight ranks staging through one socket's memory halve each other's copy rate). Read-only
    NVML query + this process's own affinity; returns the CPU count, or None when unavailable."""
    try:
        import pynvml
        pynvml.nvmlInit()
        try:
            try:      # CUDA's device order need not be NVML's: look the GPU up by its PCI address
                import torch
                pr = torch.cuda.get_device_properties(gpu_index)
                bus = f"{pr.pci_domain_id:08x}:{pr.pci_bus_id:02x}:{pr.pci_device_id:02x}.0"
                h = pynvml.nvmlDeviceGetHandleByPciBusId(bus.encode())
            except Exception:
                h = pynvml.nvmlDeviceGetHandleByIndex(gpu_index)
            words = (os.cpu_count() + 63) // 64
            mask = pynvml.nvmlDeviceGetCpuAffinity(h, words)
        finally:
            pynvml.nvmlShutdown()
        cpus = {64 * i + b for i, wd in enumerate(mask) for b in range(64) if (wd >> b) & 1}
        cpus &= os.sched_getaffinity(0)
        if not cpus:
            return None
        os.sched_setaffinity(0, cpus)
        return len(cpus)
    except Exception:
        return None


def run_gpu_arm(args):
    import torch
    import torch.distributed as dist
    from strata_b200 import ops, rope, _lib

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if not torch.cuda.is_available():
        raise SystemExit("bench.py needs a CUDA device (there is no CPU path); "
                         "use --impl reference for the CPU baseline")
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    numa_cpus = bind_to_gpu_cpus(local_rank) if world > 1 else None
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)

    C, heads, kernel = WORKLOAD["dim"], WORKLOAD["heads"], tuple(WORKLOAD["kernel"])
    D, H, W = WORKLOAD["token_grid"]
    n_tiles = WORKLOAD["tiles_per_gpu"]
    hidden = C * WORKLOAD["mlp_ratio"]
    T = D * H * W
    M = n_tiles * T

    g = torch.Generator().manual_seed(1234 + rank)
    def tn(*shape):
        w = torch.empty(*shape)
        torch.nn.init.trunc_normal_(w, std=0.02, a=-0.04, b=0.04, generator=g)
        return w
    weights = {
        "w_qkv": tn(3 * C, C), "w_proj": tn(C, C), "w_fc1": tn(hidden, C), "w_fc2": tn(C, hidden)}
    weights = {k: v.to(dev, torch.bfloat16).contiguous() for k, v in weights.items()}
    for k, n in (("b_qkv", 3 * C), ("b_proj", C), ("b_fc1", hidden), ("b_fc2", C)):
        weights[k] = torch.zeros(n, device=dev, dtype=torch.float32)
    x_host = torch.randn(n_tiles, T, C, generator=g).to(torch.bfloat16).pin_memory()
    y_host = torch.empty_like(x_host).pin_memory()
    x = x_host.to(dev)
    y = torch.empty_like(x)
    lat = (torch.linspace(0.2, 0.7, H).view(1, H, 1) - 0.3 * torch.arange(n_tiles).view(-1, 1, 1)
           ).expand(n_tiles, H, W)
    lon = (torch.linspace(0.1, 0.6, W).view(1, 1, W) + 0.7 * (torch.arange(n_tiles) + n_tiles * rank
                                                                ).view(-1, 1, 1)).expand(n_tiles, H, W)
    pos = torch.stack([lat, lon], dim=1).to(dev)
    cos, sin = rope.stereographic_rope_tables(pos, C // heads, 1, rope.default_rope_length_scale(1))
    cos, sin = cos.contiguous(), sin.contiguous()
    cs = rope.pack_rope_tables(cos, sin)
    ws = torch.empty(ops.block_workspace_bytes(M, C, hidden), dtype=torch.uint8, device=dev)

    def step(inp, out):
        ops.block_forward(inp, weights, grid=(D, H, W), num_heads=heads, kernel=kernel,
                          rope_cos=None, rope_sin=None, rope_cs=cs, workspace=ws, out=out)

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    def timed(fn, steps):
        barrier()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(steps):
            fn()
        e1.record()
        barrier()
        ms = e0.elapsed_time(e1)
        if world > 1:
            t = torch.tensor([ms], device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
        return ms

    if args.only == "pixel_stage":
        res = pixel_stage_bench(torch, dev, iters=args.steps)
        if rank == 0:
            print(json.dumps({"only": args.only, "result": res}))
        return
    if args.only == "halo_kernels":
        res = halo_kernels_bench(torch, dev, iters=args.steps)
        if rank == 0:
            print(json.dumps({"only": args.only, "result": res}))
        return
    if args.only:
        # profiling aid: run one kernel of the block alone on the bench workload
        res = kernel_breakdown(torch, ops, x, weights, cs, (D, H, W), heads, kernel, hidden,
                               iters=args.steps, only=args.only)
        if rank == 0:
            print(json.dumps({"only": args.only, "result": [
                {k: v for k, v in r.items() if k in ("name", "ms", "frac", "bound")} for r in res]}))
        return

    warm = max(args.warmup, 3)
    for _ in range(warm):
        step(x, y)
    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()
    # EXACTLY args.steps steps are timed per repeat; the region is repeated until the 20 ms
    # clock sampler has seen it for about a second (>= 10 samples under load) and the median
    # repeat is reported; a second of dense GEMMs runs into the board's power cap, so this is the
    # sustained figure (the first repeat alone, a ~50 ms burst, is reported beside it)
    repeats_ms = [timed(lambda: step(x, y), args.steps)]
    n_rep = int(min(400, max(3, 1000.0 / max(repeats_ms[0], 1e-3)))) | 1
    if world > 1:
        t = torch.tensor([n_rep], device=dev)
        dist.broadcast(t, 0)
        n_rep = int(t.item())
    for _ in range(n_rep - 1):
        repeats_ms.append(timed(lambda: step(x, y), args.steps))
    ms_total = statistics.median(repeats_ms)
    clocks = sampler.stop() if rank == 0 else None
    if clocks is not None:
        clocks["timed_repeats"] = n_rep
    status = _lib.device_status()
    ms_step = ms_total / args.steps
    tokens_job = M * world
    value = tokens_job / (ms_step * 1e-3)

    # end to end: pinned host buffers in, pinned host buffers out, through the public host API
    # (copies and compute pipelined over chunks of tiles, the same C-ABI block call inside)
    from strata_b200.host_pipeline import HostBlockPipeline
    pipe = HostBlockPipeline(T, C, hidden, device=dev, chunk_tiles=1, ring=4)
    e2e_steps = max(2, min(args.steps, 10))

    # steps are streamed: each copies its own input from pinned host memory and its own result
    # back, but a step's first host->device copy does not wait for the previous step's last
    # device->host copy; the timed region ends when the last result has landed (join)
    calls = {"n": 0}

    def e2e_step():
        calls["n"] += 1
        pipe.run(x_host, y_host, weights, grid=(D, H, W), num_heads=heads, kernel=kernel, rope_cs=cs,
                 join=calls["n"] % e2e_steps == 0)
    for _ in range(e2e_steps):
        e2e_step()
    ms_e2e = timed(e2e_step, e2e_steps) / e2e_steps
    e2e_value = tokens_job / (ms_e2e * 1e-3)

    # secondary metric: one model step over a whole tiled cubed sphere, tiles sharded over ranks
    try:
        sphere = sphere_step_bench(torch, dist, world, rank, dev, timed)
    except Exception as exc:  # reported, never fatal for the headline line
        sphere = {"error": f"{type(exc).__name__}: {exc}"[:300]}

    # secondary metric: stack of blocks over the sphere's tiles with a K/V halo exchange in
    # EVERY block (tiles sharded over ranks)
    torch.cuda.empty_cache()
    try:
        tiled = tiled_blocks_bench(torch, dist, world, rank, dev, timed)
    except Exception as exc:
        tiled = {"error": f"{type(exc).__name__}: {exc}"[:300]}
    torch.cuda.empty_cache()
    try:
        global_step = tiled_blocks_bench(torch, dist, world, rank, dev, timed, c=GLOBAL_STEP)
    except Exception as exc:
        global_step = {"error": f"{type(exc).__name__}: {exc}"[:300]}
    torch.cuda.empty_cache()

    # per-kernel breakdown (same sequence as strata_block_forward_bf16, one event pair each)
    breakdown = kernel_breakdown(torch, ops, x, weights, cs, (D, H, W), heads, kernel, hidden)
    sweep = na3d_sweep(torch, ops) if world == 1 else None
    # secondary metric: one AdaLN pixel block of the two-stage model (1 GPU; tiles are independent)
    pixel = None
    if world == 1:
        torch.cuda.empty_cache()
        try:
            pixel = pixel_stage_bench(torch, dev)
        except Exception as exc:
            pixel = {"error": f"{type(exc).__name__}: {exc}"[:300]}
        torch.cuda.empty_cache()

    if rank == 0:
        tf_peak, hbm_peak, peak_kind = measured_peaks()
        fpt = flops_per_token(C, kernel)
        dom = max(breakdown, key=lambda k: k["ms"])
        # a kernel whose arithmetic intensity lies below the machine's ridge is memory-bound
        if dom["bytes"] and dom["flop"] / dom["bytes"] < tf_peak * 1e12 / (hbm_peak * 1e9):
            dom = dict(dom, bound="hbm")
        if dom["bound"] == "tensor":
            achieved, peak, unit = dom["flop"] / (dom["ms"] * 1e-3) / 1e12, tf_peak, "TFLOP/s"
        else:
            achieved, peak, unit = dom["bytes"] / (dom["ms"] * 1e-3) / 1e9, hbm_peak, "GB/s"
        cpu_tps, cpu_ms, cores, sample = cpu_block_tokens_per_s(2, 1)
        cpu_c1 = cpu_config1_block_ms()
        cpu_halo = cpu_face_halo_ms()
        line = {
            "metric": "block_tokens_per_s", "value": value, "unit": "tokens/s", "n_gpus": world,
            "steps": args.steps, "warmup": warm, "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
            "config": WORKLOAD,
            "block_tflops": fpt * tokens_job / (ms_step * 1e-3) / 1e12,
            "block_frac_of_bf16_peak": fpt * M / (ms_step * 1e-3) / 1e12 / tf_peak,
            "block_frac_of_sustained_bf16_peak": fpt * M / (ms_step * 1e-3) / 1e12 / sustained_tflops(),
            "ms_per_step_first_repeat": repeats_ms[0] / args.steps,
            "roofline": {"kernel": dom["name"], "bound": "tensor" if dom["bound"] == "tensor" else "hbm",
                         "achieved": achieved, "peak": peak, "unit": unit, "frac": achieved / peak,
                         "peak_source": peak_kind + " (burst)", "traffic": dom.get("traffic")},
            "kernels": [{k: v for k, v in b.items() if k in ("name", "ms", "bound", "frac")}
                        for b in breakdown],
            "cpu_baseline": {"value": cpu_tps, "unit": "tokens/s", "cores": cores, "kind": "port",
                             "sample": sample},
            "e2e": {"value": e2e_value, "unit": "tokens/s", "ms_per_step": ms_e2e,
                    "h2d_bytes_per_step": x_host.numel() * 2 * world,
                    "d2h_bytes_per_step": y_host.numel() * 2 * world,
                    "cpus_per_rank": numa_cpus},
            # strong-scaling steps over the whole sphere with the halo exchange inside
            # (tiles sharded over the ranks): the 12-block encoder and the 24-block global step
            "step": tiled, "global_step": global_step,
            "sphere_step": sphere, "na3d_sweep": sweep, "pixel_stage": pixel,
            "cpu_baseline_config1": cpu_c1, "cpu_baseline_face_halo": cpu_halo,
            "gpu_launches": 7 * args.steps, "device_status": status, "clocks": clocks,
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


SPHERE = dict(faces=6, face_tokens=128, tile_tokens=64, halo_tokens=8, depth=16, dim=512, heads=8,
              kernel=[3, 9, 9], blocks=2, channels=8)


def sphere_step_bench(torch, dist, world, rank, dev, timed, steps=3):
    """Strong-scaling companion metric: halo exchange (peer memory) + 2-block backbone on the
    padded tiles + crop, for 24 tiles of 16x64x64 tokens with an 8-token halo."""
    from strata_b200.rollout import TiledSphereStepper
    from strata_b200.topology import TileTopology
    from strata_b200.wrappers import StrataBackboneModel
    c = SPHERE
    topo = TileTopology(world, rank, c["face_tokens"], c["tile_tokens"], c["halo_tokens"])
    P = topo.padded_tile_size
    torch.manual_seed(7)
    net = StrataBackboneModel(depth=c["depth"], height=P, width=P, n_layers=c["blocks"], patch_size=1,
                              in_chans=c["channels"], base_out_chans=c["channels"],
                              embed_dim=c["dim"], num_heads=c["heads"], attn_kernel=tuple(c["kernel"]),
                              do_rope_2d_stereographic=True, index_is_latlon=True,
                              do_bf16_mixed=True).to(dev).eval()
    stepper = TiledSphereStepper(net, topo, device=dev)
    g = torch.Generator(device=dev).manual_seed(100 + rank)
    x = torch.randn(c["channels"], c["depth"], topo.tiles_per_rank, c["tile_tokens"], c["tile_tokens"],
                    device=dev, generator=g)
    state = {"x": x}

    def step():
        state["x"] = stepper(state["x"]).clamp_(-10, 10)
    for _ in range(2):
        step()
    ms = timed(step, steps) / steps
    stepper.halo.check_status()
    # halo exchange alone
    ms_halo = timed(lambda: stepper.halo(x), 5) / 5
    halo_bytes = x.numel() // (c["tile_tokens"] ** 2) * (P * P + c["tile_tokens"] ** 2) * 4
    # windowed overlap-add un-pad of the padded outputs (alternative to the crop)
    from strata_b200.halo import NormalizedCopyHaloAdjoint, kbd_window
    unpad = NormalizedCopyHaloAdjoint(stepper.halo, window=kbd_window(P))
    ypad = stepper.halo(x)
    for _ in range(2):      # the first call grows the peer buffer to the padded size (an IPC exchange)
        unpad(ypad)
    ms_unpad = timed(lambda: unpad(ypad), 5) / 5
    out = dict(ms_per_step=ms, halo_ms=ms_halo, halo_gbs=halo_bytes / (ms_halo * 1e-3) / 1e9,
               unpad_adjoint_ms=ms_unpad, unpad_adjoint_gbs=halo_bytes / (ms_unpad * 1e-3) / 1e9,
               scaling="strong", config=c, tiles_per_rank=topo.tiles_per_rank,
               padded_tokens_per_step=topo.total_tiles * c["depth"] * P * P)
    stepper.close()
    del stepper, net
    torch.cuda.empty_cache()
    return out


TILED = dict(name="c3", faces=6, face_tokens=256, tile_tokens=128, halo_tokens=8, depth=16, dim=768,
             heads=12, kernel=[5, 13, 13], blocks=12, mlp_ratio=4, rollout_steps=1)
# the global cubed-sphere step: 6 faces of 16 x 256 x 256 tokens = 96 tiles of 64 x 64 with a
# 16-token halo, 24 blocks of dim 1024 / 16 heads. The kernel is not stated by the benchmark
# configuration; (3, 9, 9) - the single-block configuration's - is used. The step runs in token
# space (the patch embedding of the 2048 x 2048 x 128 fields is outside the block path).
GLOBAL_STEP = dict(name="c5", faces=6, face_tokens=256, tile_tokens=64, halo_tokens=16, depth=16, dim=1024,
                   heads=16, kernel=[3, 9, 9], blocks=24, mlp_ratio=4, rollout_steps=10)


def tiled_blocks_bench(torch, dist, world, rank, dev, timed, c=None, steps=None):
    """Strong-scaling step: a stack of blocks over all tiles of the sphere (sharded over the ranks
    as the reference's TileTopology does) with a K/V halo exchanged through peer memory in EVERY
    block, run as a rollout (each step's tokens are the next step's input). Reports the time of
    one step (max over ranks), its algorithmic TFLOP/s and the exchange alone."""
    import numpy as np
    from strata_b200.halo_block import TiledBlockRunner
    from strata_b200.rollout import equiangular_cubed_sphere_latlon
    from strata_b200.topology import TileTopology
    c = TILED if c is None else c
    face, T, C = c["face_tokens"], c["tile_tokens"], c["dim"]
    topo = TileTopology(world, rank, face, T, c["halo_tokens"])
    lat, lon = equiangular_cubed_sphere_latlon(face)
    full = TileTopology(1, 0, face, T, 0)
    cut = lambda g: np.stack([g[f, i * T:(i + 1) * T, j * T:(j + 1) * T] for f, i, j in full.global_tiles])
    lat, lon = cut(lat), cut(lon)
    gen = torch.Generator().manual_seed(4321)
    hidden = C * c["mlp_ratio"]

    def tn(*shape):
        w = torch.empty(*shape)
        torch.nn.init.trunc_normal_(w, std=0.02, a=-0.04, b=0.04, generator=gen)
        return w.to(dev, torch.bfloat16)
    blocks = []
    for _ in range(c["blocks"]):
        w = {"w_qkv": tn(3 * C, C), "w_proj": tn(C, C), "w_fc1": tn(hidden, C), "w_fc2": tn(C, hidden)}
        for k, n in (("b_qkv", 3 * C), ("b_proj", C), ("b_fc1", hidden), ("b_fc2", C)):
            w[k] = torch.zeros(n, device=dev, dtype=torch.float32)
        blocks.append(w)
    tokens = c["depth"] * T * T
    g = torch.Generator(device=dev).manual_seed(200 + rank)
    state = {"x": torch.randn(topo.tiles_per_rank, tokens, C, device=dev, generator=g).bfloat16()}
    run = TiledBlockRunner(topo, depth=c["depth"], dim=C, num_heads=c["heads"],
                           kernel=tuple(c["kernel"]), lat_deg=lat, lon_deg=lon,
                           rope_length_scale=float(np.radians(90.0 / face)), device=dev)

    def step():
        y = state["x"]
        for w in blocks:
            y = run.block_forward(y, w)
        state["x"] = y
    # a single GPU holds all the tiles: it times fewer steps of the rollout (the step time is
    # what is reported)
    n_steps = steps if steps is not None else (c["rollout_steps"] if world >= 4 else min(2, c["rollout_steps"]))
    step()
    ms = timed(step, n_steps) / n_steps
    run.check_status()
    out = {"config": c["name"], "ms_per_step": ms, "rollout_steps_timed": n_steps}
    qkv, ptrs = run._slot(run._epoch)

    def exchange():       # the exchange alone (barrier + K/V gather of one block)
        run._epoch += 1
        run._exchange(qkv, ptrs)
    exchange()
    out["exchange_ms_per_block"] = timed(exchange, 5) / 5
    P = topo.padded_tile_size
    halo_cells = topo.tiles_per_rank * c["depth"] * (P * P - T * T)
    out["exchange_bytes_per_block"] = halo_cells * 2 * C * 2 * 2   # K,V read + written
    run.close()
    del run, blocks, state
    torch.cuda.empty_cache()
    total_tokens = topo.total_tiles * tokens
    out.update(tokens_per_s=total_tokens / (ms * 1e-3), scaling="strong", workload=c,
               tiles_per_rank=topo.tiles_per_rank,
               tflops=flops_per_token(C, tuple(c["kernel"])) * total_tokens * c["blocks"] / (ms * 1e-3) / 1e12)
    return out


NA_SWEEP = dict(B=8, D=32, H=96, W=96, heads=16, head_dim=64, kernels=[[3, 7, 7], [3, 13, 13], [5, 15, 15]])


def na3d_sweep(torch, ops, iters=3):
    """Standalone neighbourhood attention on Q/K/V [8, 32, 96, 96, 16, 64] for three kernels:
    milliseconds per launch, algorithmic TFLOP/s (4 * window * head_dim per query and head) and
    algorithmic GB/s (q, k, v read and o written once: the bound of the smallest kernel, whose
    arithmetic intensity lies below the ridge of the machine)."""
    c = NA_SWEEP
    shape = (c["B"], c["D"], c["H"], c["W"], c["heads"], c["head_dim"])
    try:
        q, k, v = (torch.randn(shape, device="cuda").bfloat16() for _ in range(3))
        o = torch.empty_like(q)
        res = []
        for kern in c["kernels"]:
            for _ in range(2):
                ops.na3d(q, k, v, tuple(kern), out=o)
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(iters):
                ops.na3d(q, k, v, tuple(kern), out=o)
            e1.record()
            torch.cuda.synchronize()
            ms = e0.elapsed_time(e1) / iters
            flop = 4.0 * kern[0] * kern[1] * kern[2] * c["head_dim"] * q.numel() / c["head_dim"]
            res.append({"kernel": kern, "ms": ms, "tflops": flop / (ms * 1e-3) / 1e12,
                        "gbs": 4 * q.numel() * 2 / (ms * 1e-3) / 1e9})
        del q, k, v, o
        torch.cuda.empty_cache()
        return {"shape": list(shape), "results": res}
    except Exception as exc:
        return {"error": f"{type(exc).__name__}: {exc}"[:300]}


def halo_kernels_bench(torch, dev, iters=5):
    """Times the memory-bound kernels around the block on one GPU (all sources local): field and
    token halo gathers, the per-block K/V halo gather, the overlap-add un-pad and the fused
    pre-/post-processing, each with its algorithmic bytes (payload read once + written once) and
    the fraction of the measured copy bandwidth. Sizes (kept to a few GB so that the same
    command can run under ncu): 24 tiles of 64x64 cells with a halo of 8, 8 levels, 768 channels
    in token space, 64 field channels."""
    import ctypes
    import numpy as np
    from strata_b200 import _lib, ops
    from strata_b200.halo import DistributedTileCopyHaloPadding, NormalizedCopyHaloAdjoint, kbd_window
    from strata_b200.halo_block import TiledBlockRunner
    from strata_b200.rollout import equiangular_cubed_sphere_latlon
    from strata_b200.topology import TileTopology
    _, hbm_peak, _ = measured_peaks()
    face, T, h, D, C, CF = 128, 64, 8, 8, 768, 64
    topo = TileTopology(1, 0, face, T, h)
    P, tpr = topo.padded_tile_size, topo.tiles_per_rank
    pad = DistributedTileCopyHaloPadding(topology=topo, device=dev)
    unpad = NormalizedCopyHaloAdjoint(pad, window=kbd_window(P))
    fields = torch.randn(CF, D, tpr, T, T, device=dev)
    padded = pad(fields)
    lat, lon = equiangular_cubed_sphere_latlon(face)
    full = TileTopology(1, 0, face, T, 0)
    cut = lambda g: np.stack([g[f, i * T:(i + 1) * T, j * T:(j + 1) * T] for f, i, j in full.global_tiles])
    run = TiledBlockRunner(topo, depth=D, dim=C, num_heads=C // 64, kernel=(5, 13, 13),
                           lat_deg=cut(lat), lon_deg=cut(lon),
                           rope_length_scale=float(np.radians(90.0 / face)), device=dev)
    qkv, ptrs = run._slot(1)
    x5 = torch.randn(tpr, 13, D, P, P, device=dev)
    latp = torch.rand(tpr, P, P, device=dev)
    lat0 = torch.rand(tpr, device=dev)
    a_mat = ops.preprocess_patches(x5, latp, latp, lat0, lat0, wind=(0, 1), concat_lat=True)
    ymat = torch.randn(tpr * D * P * P, 16, device=dev).bfloat16()

    def exchange():
        run._epoch += 1
        run._exchange(qkv, ptrs)
    halo_cells = tpr * D * (P * P - T * T)
    items = [
        ("halo_gather_fields", lambda: pad(fields), fields.numel() * 4 + padded.numel() * 4),
        ("halo_adjoint_fields", lambda: unpad(padded), fields.numel() * 4 + padded.numel() * 4),
        ("halo_gather_kv", exchange, halo_cells * 2 * C * 2 * 2),
        ("preprocess_patches", lambda: ops.preprocess_patches(x5, latp, latp, lat0, lat0, wind=(0, 1),
                                                              concat_lat=True),
         x5.numel() * 4 + a_mat.numel() * 2),
        ("postprocess_fields", lambda: ops.postprocess_fields(ymat, (tpr, 13, D, P, P), latp, latp,
                                                              lat0, lat0, wind=(0, 1)),
         ymat.shape[0] * 13 * 2 + tpr * 13 * D * P * P * 4),
    ]
    out = []
    for name, fn, nbytes in items:
        fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(iters):
            fn()
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / iters
        out.append({"name": name, "ms": ms, "gbs": nbytes / (ms * 1e-3) / 1e9,
                    "frac_of_hbm": nbytes / (ms * 1e-3) / 1e9 / hbm_peak})
    run.close()
    return out


PIXEL = dict(depth=24, height=256, width=256, patch=4, backbone_dim=1024, dim=128, heads=2,
             kernel=(9, 9, 9), qk_norm=True)


def pixel_stage_bench(torch, dev, iters=3):
    """One AdaLN pixel block of the two-stage model at the production channel widths (backbone
    1024, pixel 128, 2 heads, 9x9x9 attention, bilinear_dw conditioning) on one 24 x 256 x 256
    pixel tile (1.57 M pixel tokens, 98 k backbone tokens): every kernel of the block alone, with
    its algorithmic bytes or flops, then the whole block (modulation + forward)."""
    from strata_b200 import _lib, ops
    from strata_b200.ops import EPI_GELU
    from strata_b200.pixel import StrataPixel3DBlock
    tf_peak, hbm_peak, _ = measured_peaks()
    c = PIXEL
    D, H, W, f, Cb, C = c["depth"], c["height"], c["width"], c["patch"], c["backbone_dim"], c["dim"]
    M = D * H * W
    torch.manual_seed(0)
    blk = StrataPixel3DBlock(C, c["heads"], 4.0, c["qk_norm"], False, c["kernel"], Cb, adaln=True)
    blk.mlp.layers[1].approximate = "tanh"
    with torch.no_grad():
        blk.adaln_bilinear_dw_proj.weight.normal_(0, 0.5 / Cb ** 0.5)
    blk = blk.to(dev).eval()
    wts = blk.device_weights()
    s = torch.randn(1, D, H // f, W // f, Cb, device=dev).bfloat16()
    x = torch.randn(M, C, device=dev).bfloat16()
    n = min(M, 1 << 18)
    cond = torch.empty(n, Cb, device=dev, dtype=torch.bfloat16)
    with torch.inference_mode():
        mod = blk.modulation(s, f)
        sl = lambda i: mod[:, i * C:(i + 1) * C]
        xn = ops.adaln_rows(x, shift=sl(0), scale=sl(1))
        qkv = ops.linear(xn, wts["w_qkv"], wts["b_qkv"])
        q6 = qkv.view(1, D, H, W, 3, c["heads"], 64)
        attn = ops.na3d(q6[:, :, :, :, 0], q6[:, :, :, :, 1], q6[:, :, :, :, 2], c["kernel"]).view(-1, C)
        h = ops.linear(xn, wts["w_fc1"], wts["b_fc1"], EPI_GELU)
        y = ops.linear(attn, wts["w_proj"], wts["b_proj"])
        hidden, z = wts["w_fc1"].shape[0], torch.empty_like(x)
        kd, kh, kw = c["kernel"]

        def mlp_kernel():                       # as a model's call launches it
            g = sl(5)
            _lib.check(_lib.load().strata_mlp_bf16(
                xn.data_ptr(), C, wts["w_fc1"].data_ptr(), wts["b_fc1"].data_ptr(), wts["w_fc2"].data_ptr(),
                wts["b_fc2"].data_ptr(), x.data_ptr(), C, g.data_ptr(), g.stride(0), z.data_ptr(), C, M, C, hidden,
                _lib.stream_of(x)), "strata_mlp_bf16")
        items = [
            ("adaln_cond (2^18 pixels)", lambda: ops.adaln_cond(s, wts["w_dw"], wts["b_dw"], f, 0, n, out=cond),
             "hbm", n * Cb * 2),
            ("modulation GEMM (2^18 pixels)", lambda: ops.linear(cond, wts["w_mod"], wts["b_mod"], out=mod[:n]),
             "tensor", 2.0 * n * Cb * 6 * C),
            ("ln_modulate", lambda: ops.adaln_rows(x, shift=sl(0), scale=sl(1)), "hbm", M * C * 2 * 4),
            ("qkv GEMM + q/k norm", lambda: ops.qkv_rope(xn, wts["w_qkv"], wts["b_qkv"], 64, None, None,
                                                         D * H * W, H * W, qk_norm=True), "hbm", M * C * 2 * 4),
            ("na3d 9x9x9", lambda: ops.na3d(q6[:, :, :, :, 0], q6[:, :, :, :, 1], q6[:, :, :, :, 2],
                                             c["kernel"]), "tensor", 4.0 * M * C * kd * kh * kw),
            ("proj GEMM", lambda: ops.linear(attn, wts["w_proj"], wts["b_proj"], out=y), "hbm", M * C * 2 * 2),
            ("gated residual + ln_modulate", lambda: ops.adaln_rows(x, y=y, gate=sl(2), shift=sl(3), scale=sl(4)),
             "hbm", M * C * 2 * 7),
            ("MLP kernel: fc1, GELU, fc2, gated residual", mlp_kernel, "tensor", 4.0 * M * C * hidden),
            # a block called as a module (hooks, replaced blocks) takes these three for the MLP kernel
            ("fc1 GEMM + GELU (module)", lambda: ops.linear(xn, wts["w_fc1"], wts["b_fc1"], EPI_GELU, out=h),
             "hbm", M * C * 2 * 5),
            ("fc2 GEMM (module)", lambda: ops.linear(h, wts["w_fc2"], wts["b_fc2"], out=y), "hbm", M * C * 2 * 5),
            ("gated residual (module)", lambda: ops.adaln_rows(x, y=y, gate=sl(5), norm=False), "hbm",
             M * C * 2 * 4),
            ("whole block as a module (modulation + forward)", lambda: blk(x, (D, H, W), blk.modulation(s, f), 1),
             None, 0),
        ]
        out = []
        for name, fn, bound, work in items:
            fn()
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(iters):
                fn()
            e1.record()
            torch.cuda.synchronize()
            ms = e0.elapsed_time(e1) / iters
            r = {"name": name, "ms": ms}
            if bound == "hbm":
                r.update(bound="hbm", gbs=work / (ms * 1e-3) / 1e9,
                         frac=work / (ms * 1e-3) / 1e9 / hbm_peak)
            elif bound == "tensor":
                r.update(bound="tensor", tflops=work / (ms * 1e-3) / 1e12,
                         frac=work / (ms * 1e-3) / 1e12 / tf_peak)
            else:
                r.update(pixel_tokens_per_s=M / (ms * 1e-3))
            out.append(r)
    return {"config": {k: (list(v) if isinstance(v, tuple) else v) for k, v in c.items()},
            "pixel_tokens": M, "kernels": out}


def kernel_breakdown(torch, ops, x, weights, cs, grid, heads, kernel, hidden, iters=5,
                     only=None):
    """Times each kernel of the block alone (CUDA events on the launching stream) and attaches
    its algorithmic flops / bytes and roofline fraction."""
    tf_peak, hbm_peak, _ = measured_peaks()
    D, H, W = grid
    n_tiles, T, C = x.shape
    M = n_tiles * T
    x2 = x.reshape(M, C)
    xn = ops.layernorm(x2)
    qkv = ops.qkv_rope(xn, weights["w_qkv"], weights["b_qkv"], C // heads, None, None, T, H * W,
                       rope_cs=cs)
    q6 = qkv.view(n_tiles, D, H, W, 3, heads, C // heads)
    attn = torch.empty(n_tiles, D, H, W, heads, C // heads, dtype=torch.bfloat16, device=x.device)
    x1 = torch.empty_like(x2)
    hbuf = torch.empty(M, hidden, dtype=torch.bfloat16, device=x.device)
    y = torch.empty_like(x2)
    K = kernel[0] * kernel[1] * kernel[2]
    items = [
        ("layernorm_rows", lambda: ops.layernorm(x2), "hbm", 0, 4 * M * C),
        ("gemm_qkv_rope", lambda: ops.qkv_rope(xn, weights["w_qkv"], weights["b_qkv"], C // heads,
                                               None, None, T, H * W, rope_cs=cs), "tensor",
         6 * C * C * M, 8 * M * C),
        ("na3d_fwd", lambda: ops.na3d(q6[..., 0, :, :], q6[..., 1, :, :], q6[..., 2, :, :], kernel,
                                      out=attn), "tensor", 4 * K * C * M, 8 * M * C),
        ("gemm_proj_residual", lambda: ops.linear(attn.view(M, C), weights["w_proj"], weights["b_proj"],
                                                  ops.EPI_RESIDUAL, x2, out=x1), "tensor",
         2 * C * C * M, 6 * M * C),
        ("gemm_fc1_gelu", lambda: ops.linear(xn, weights["w_fc1"], weights["b_fc1"], ops.EPI_GELU,
                                             out=hbuf), "tensor", 2 * C * hidden * M, 2 * M * (C + hidden)),
        ("gemm_fc2_residual", lambda: ops.linear(hbuf, weights["w_fc2"], weights["b_fc2"],
                                                 ops.EPI_RESIDUAL, x1, out=y), "tensor",
         2 * C * hidden * M, 2 * M * (hidden + 2 * C)),
    ]
    out = []
    for name, fn, bound, flop, nbytes in items:
        if only is not None and name != only:
            continue
        fn()
        torch.cuda.synchronize()
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(iters):
            fn()
        e1.record()
        torch.cuda.synchronize()
        ms = e0.elapsed_time(e1) / iters
        frac = (flop / (ms * 1e-3) / 1e12 / tf_peak) if bound == "tensor" else (
            nbytes / (ms * 1e-3) / 1e9 / hbm_peak)
        out.append({"name": name, "ms": ms, "bound": bound, "flop": flop, "bytes": nbytes,
                    "frac": frac, "traffic": NCU_TRAFFIC_BYTES.get(name)})
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="strata_b200", choices=["strata_b200", "reference"])
    ap.add_argument("--only", default=None,
                    help="run a single kernel of the block (name as in the 'kernels' list) "
                         "--steps times and print its time; used for ncu captures")
    args = ap.parse_args()
    if args.impl == "reference":
        run_reference_arm(args)
        return
    # Libraries may print to stdout (NCCL prints a version banner there): while the benchmark
    # runs, file descriptor 1 points at stderr, and the one JSON line goes to the real stdout.
    sys.stdout.flush()
    real_stdout = os.dup(1)
    os.dup2(2, 1)
    sys.stdout = os.fdopen(real_stdout, "w", buffering=1)
    run_gpu_arm(args)
    sys.stdout.flush()


if __name__ == "__main__":
    main()
