"""Headline benchmark: fused all_gather_matmul at the Llama-3-70B TP shape.

    python bench.py --gpus N --steps K --warmup W            (N = 1)
    python -m torch.distributed.run --nnodes=1 --nproc-per-node N \
        --master-addr 127.0.0.1 --master-port P bench.py --gpus N --steps K --warmup W

Metric: aggregate TFLOPS of `all_gather_matmul` over the N GPUs.  M = 16384
gathered rows (each rank holds A shard [16384/N, 8192] in symmetric memory),
B = [3584, 8192] per rank, C = [16384, 3584] per rank, bf16, values N(0, 0.02),
seeded per rank.  Every rank computes the full 0.962 TFLOP product, so per-GPU
work is fixed as N grows ("weak").  At N = 8 this is the configuration behind
the upstream table row README.md:29 (fused 1846 µs on 8xH100 = 521 TFLOPS per
GPU); `vs_baseline` is TFLOPS per GPU divided by that.

Timing: W untimed steps, then K steps, each bracketed by CUDA events on the
launching stream with an L2 flush (256 MB write) before it; barrier +
synchronize on both sides of the timed region; maximum over ranks.
`e2e` repeats the measurement through the public API including, every step,
the host-to-device copy of the step's A shard from pinned memory and a
device-to-host read of a checksum of C.  `same_box_baseline` is the library
composition (NCCL all-gather + cuBLAS) timed the same way in the same run.
`e2e` is that step fed the way a serving loop feeds it: two shard buffers, the
next step's host-to-device copy on a copy stream under the current step's
kernel; `e2e_serial` is the same step with copy, kernel and read-back strictly
one after the other.

At N > 1 the line also carries the other half of the metric (extra keys, each
gated by its own check against NCCL): `all_reduce` (µs and bus GB/s at 4 KiB,
64 KiB, 1 MiB and 64 MiB for `all_reduce(auto)`, `one_shot_all_reduce`, NCCL and
the upstream Triton one-shot kernel, unmodified, where it loads) and
`gemv_all_reduce` (fused GEMV + all-reduce against cuBLAS + NCCL at batch 1, 4
and 16, Llama-3-70B down-projection shard).  `--no-extras` leaves them out.
"""
from __future__ import annotations

import argparse
import json
import os
import sys
import time

import torch
import torch.distributed as dist

M_TOTAL, N_PER_RANK, K_DIM = 16384, 3584, 8192
PUBLISHED_FUSED_US_H100 = 1846.0   # upstream README.md:29
PUBLISHED_TFLOPS_PER_GPU = 2.0 * M_TOTAL * N_PER_RANK * K_DIM / PUBLISHED_FUSED_US_H100 / 1e6


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-extras", action="store_true",
                    help="N > 1: skip the all-reduce and GEMV + all-reduce sections")
    return ap.parse_args()


def all_reduce_section(world, rank, dev):
    """µs (device time, maximum over ranks) and bus GB/s of the all-reduce kernels at four sizes,
    beside NCCL and the upstream Triton kernel on the same box.  Graph replay up to 1 MiB (the
    eager number would be CPU launch cost), CUDA events at 64 MiB."""
    import symm_mem_recipes_b200 as smr
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.benchmark import benchmark_with_event, benchmark_with_graph

    sizes = [4096, 65536, 1 << 20, 64 << 20]
    buf = symm_mem.empty(sizes[-1] // 2, dtype=torch.bfloat16, device=dev)
    hdl = symm_mem.rendezvous(buf)
    torch.manual_seed(1234 + rank)
    plain = torch.randn(sizes[-1] // 2, device=dev).to(torch.bfloat16)
    ref_fn = ref_buf = None
    ref_note = None
    try:
        sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
        from baseline.reference_triton import load_reference_one_shot
        ref_fn, ref_alloc = load_reference_one_shot()
        ref_buf = ref_alloc((8 << 20) // 2, dev)
        ref_buf.normal_()
    except Exception as e:  # noqa: BLE001 - the section goes on without that column
        ref_fn, ref_note = None, f"{type(e).__name__}: {e}"
    out = {"unit": "us", "bus_gbs": "2 (N-1)/N * bytes / time", "sizes": {}}
    if ref_note:
        out["reference_triton_unavailable"] = ref_note
    for nbytes in sizes:
        numel = nbytes // 2
        t = buf[:numel]
        # check: the dispatcher's result against NCCL on the same input
        t.copy_(plain[:numel])
        want = plain[:numel].clone()
        dist.all_reduce(want)
        hdl.barrier()
        smr.all_reduce(t)
        hdl.barrier()
        symm_mem.check_status(dev)
        scale = float(want.float().abs().max()) or 1.0
        err = float((t.float() - want.float()).abs().max()) / scale
        ok = max_all(0.0 if err < 2e-2 else 1.0, dev) == 0.0
        t.copy_(plain[:numel])
        hdl.barrier()
        one_out = torch.empty_like(t)
        impls = {"auto": lambda: smr.all_reduce(t), "nccl": lambda: dist.all_reduce(plain[:numel])}
        if nbytes <= (8 << 20):
            impls["one_shot"] = lambda: smr.one_shot_all_reduce(t, out=one_out)
            if ref_fn is not None:
                rt = ref_buf[:numel]
                impls["reference_triton"] = lambda: ref_fn(rt)
        row = {"matches_nccl": ok, "algo": smr.ops.choose_algo(nbytes, world, hdl.has_multicast)}
        for name, fn in impls.items():
            if nbytes <= (4 << 20):
                us = benchmark_with_graph(fn, calls_per_graph=20, warmup_iters=5, replays=10)
            else:
                us = benchmark_with_event(fn, 5, 20, flush_l2=False)
            row[name] = {"us": round(us, 2), "bus_gbs": round(2 * (world - 1) / world * nbytes / us / 1e3, 1)}
            buf.normal_()
            plain.normal_()
        symm_mem.check_status(dev)
        out["sizes"][str(nbytes)] = row
    return out


def gemv_section(world, rank, dev):
    """Fused GEMV + all-reduce against cuBLAS + NCCL at the Llama-3-70B down-projection decode
    shape (x [b, 3584], W [3584, 8192] per rank), device time per call from graph replay over
    four weight copies (224 MB, more than the L2 holds), maximum over ranks."""
    import symm_mem_recipes_b200 as smr
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.benchmark import benchmark_with_graph

    K, N = 3584, 8192
    torch.manual_seed(77 + rank)
    weights = [(torch.randn(K, N, device=dev) * 0.02).to(torch.bfloat16) for _ in range(4)]
    out = {"unit": "us", "shape": {"K_per_rank": K, "N": N}, "batches": {}}
    for b in (1, 4, 16):
        x = (torch.randn(b, K, device=dev) * 0.02).to(torch.bfloat16)
        y = torch.empty(b, N, dtype=torch.bfloat16, device=dev)
        smr.gemv_all_reduce(x, weights[0], y)
        symm_mem.check_status(dev)
        want = smr.reference_gemv_all_reduce(x, weights[0])
        ok = bool(torch.allclose(y.float(), want.float(), rtol=2e-2, atol=2e-2))
        ok = max_all(0.0 if ok else 1.0, dev) == 0.0
        state = {"i": 0}

        def fused():
            state["i"] = (state["i"] + 1) % 4
            smr.gemv_all_reduce(x, weights[state["i"]], y)

        def lib():
            state["i"] = (state["i"] + 1) % 4
            smr.reference_gemv_all_reduce(x, weights[state["i"]])

        us = benchmark_with_graph(fused, calls_per_graph=20, replays=10)
        us_lib = benchmark_with_graph(lib, calls_per_graph=20, replays=10)
        symm_mem.check_status(dev)
        out["batches"][str(b)] = {"matches_library": ok, "fused_us": round(us, 2),
                                  "cublas_plus_nccl_us": round(us_lib, 2), "speedup": round(us_lib / us, 3)}
    return out


def max_all(value, dev):
    from symm_mem_recipes_b200.utils.benchmark import max_over_ranks
    return max_over_ranks(value, dev)


def reference_arm(args) -> int:
    """The upstream package installs into baseline/_ref, but its all-gather
    matmul module cannot be imported with the Triton of this image."""
    root = os.path.dirname(os.path.abspath(__file__))
    ref = os.path.join(root, "baseline", "_ref")
    rank = int(os.environ.get("RANK", "0"))
    reason = None
    if not os.path.isdir(os.path.join(ref, "symm_mem_recipes")):
        reason = "baseline/_ref is not installed"
    else:
        sys.path.insert(0, ref)
        try:
            import symm_mem_recipes.triton_all_gather_matmul  # noqa: F401
            reason = ("reference imported, but its fused kernel needs tl._experimental_descriptor_load "
                      "and the 2-argument stream_write_value32, both absent from this image")
        except Exception as e:  # noqa: BLE001
            reason = (f"unmodified reference cannot be imported on this image: {type(e).__name__}: {e} "
                      "(symm_mem_recipes/triton_all_gather_matmul.py:8 uses a Triton API removed before 3.6)")
    line = {"impl": "reference", "unavailable": reason}
    world = int(os.environ.get("WORLD_SIZE", "1"))
    if world > 1:
        # The all-reduce half of the metric does run unmodified on this image (with a stub for the
        # missing `expecttest` module): upstream's own kernel, wrapper and timing helper
        # (symm_mem_recipes/triton_one_shot_all_reduce.py:96-125, 156-160), at four message sizes.
        try:
            line["all_reduce"] = reference_all_reduce(world, rank)
        except Exception as e:  # noqa: BLE001
            line["all_reduce"] = {"unavailable": f"{type(e).__name__}: {e}"}
    if rank == 0:
        print(json.dumps(line))
    return 0


def reference_all_reduce(world, rank):
    """Median kernel time (µs, rank 0, torch.profiler) of upstream's one-shot all-reduce on torch's
    own symmetric memory, measured with upstream's `benchmark_with_profiler` as its driver does."""
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
    dist.init_process_group("nccl", device_id=dev)
    try:
        sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
        from baseline.reference_triton import load_reference_one_shot
        one_shot, alloc = load_reference_one_shot()
        from symm_mem_recipes.utils import benchmark_with_profiler
        sizes = [4096, 65536, 1 << 20, 8 << 20]
        buf = alloc(sizes[-1] // 2, dev)
        buf.fill_(1)
        res = {"unit": "us", "how": "upstream one_shot_all_reduce timed by upstream benchmark_with_profiler "
                                    "(median kernel time on rank 0, 200 iterations)", "sizes": {}}
        ok = bool(one_shot(buf[:8192]).eq(world).all())           # upstream's own check (:153-154)
        res["output_equals_world_size"] = ok
        for nbytes in sizes:
            t = buf[:nbytes // 2]
            us = benchmark_with_profiler(lambda: one_shot(t), "one_shot_all_reduce_kernel", benchmark_iters=200)
            res["sizes"][str(nbytes)] = {"us": round(float(us), 2),
                                         "bus_gbs": round(2 * (world - 1) / world * nbytes / us / 1e3, 1) if us else None}
        return res
    finally:
        torch.cuda.synchronize()
        dist.barrier()
        dist.destroy_process_group()


def main() -> int:
    args = parse_args()
    if args.impl == "reference":
        return reference_arm(args)

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if world != args.gpus:
        if world == 1 and args.gpus > 1:
            raise SystemExit("launch with torch.distributed.run --nproc-per-node N for --gpus N > 1")
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    distributed = world > 1
    if distributed:
        os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
        dist.init_process_group("nccl", device_id=dev)

    import symm_mem_recipes_b200 as smr
    from symm_mem_recipes_b200._ext import C
    from symm_mem_recipes_b200.ops.ag_matmul import _num_sms
    from symm_mem_recipes_b200.parallel import symm_mem
    from symm_mem_recipes_b200.utils.benchmark import ClockSampler, flush_l2, max_over_ranks

    rows = M_TOTAL // world
    sms = _num_sms(dev) if dev.type == "cuda" else 148
    torch.manual_seed(42 + rank)
    a_shard = symm_mem.empty(rows, K_DIM, dtype=torch.bfloat16, device=dev)
    a_host = (torch.randn(rows, K_DIM) * 0.02).to(torch.bfloat16).pin_memory()
    a_shard.copy_(a_host)
    b = (torch.randn(N_PER_RANK, K_DIM, device=dev) * 0.02).to(torch.bfloat16)
    # the gathered A is a side output only when there is something to gather
    a_out = symm_mem.empty(M_TOTAL, K_DIM, dtype=torch.bfloat16, device=dev) if world > 1 else None
    c_out = torch.empty(M_TOTAL, N_PER_RANK, dtype=torch.bfloat16, device=dev)
    if distributed:
        symm_mem.rendezvous(a_shard)
        symm_mem.rendezvous(a_out)
    checksum_host = torch.empty(1, dtype=torch.float32).pin_memory()

    def step():
        smr.all_gather_matmul(a_shard, b, a_out, c_out)

    def sync_all():
        torch.cuda.synchronize()
        if distributed:
            dist.barrier()
        torch.cuda.synchronize()

    # correctness gate before timing: compare with the library composition
    step()
    symm_mem.check_status(dev)
    if distributed:
        ref = smr.reference_all_gather_matmul(a_shard, b)
    else:
        ref = torch.matmul(a_shard, b.t())
    ok = bool(torch.allclose(c_out.float(), ref.float(), rtol=2e-2, atol=2e-3))
    del ref
    # every rank learns the outcome (a rank that left alone would strand the others in a collective)
    if max_over_ranks(0.0 if ok else 1.0, dev) != 0.0:
        raise SystemExit(f"rank {rank}: fused result differs from all-gather + matmul (this rank ok: {ok})")

    flops = 2.0 * M_TOTAL * N_PER_RANK * K_DIM

    def timed(fn, steps):
        begins = [torch.cuda.Event(enable_timing=True) for _ in range(steps)]
        ends = [torch.cuda.Event(enable_timing=True) for _ in range(steps)]
        sync_all()
        t0 = time.perf_counter()
        for i in range(steps):
            flush_l2(dev)
            begins[i].record()
            fn()
            ends[i].record()
        sync_all()
        wall = time.perf_counter() - t0
        ms = sum(b_.elapsed_time(e_) for b_, e_ in zip(begins, ends)) / steps
        return max_over_ranks(ms, dev), wall

    # nvidia-smi needs a moment to start: the sampler runs from the warm-up on, and after the
    # reported measurement the same timed region is repeated (not reported) for about a second so
    # that the sampler sees the GPU under this load.  The repeat count is derived from the
    # max-over-ranks time, hence identical on every rank: the region contains collectives.
    # ---- the library composition on the same box, same shape, same timing: NCCL all-gather + cuBLAS
    #      (upstream's own baseline, triton_all_gather_matmul.py:322-326); cuBLAS alone when N = 1 ----
    def baseline_step():
        if distributed:
            smr.reference_all_gather_matmul(a_shard, b)
        else:
            torch.matmul(a_shard, b.t(), out=c_out)

    with ClockSampler(local_rank, period_ms=50) as clocks:
        for _ in range(max(args.warmup, 3)):
            step()
        ms_per_step, wall = timed(step, args.steps)
        # the baseline right after it, with the same warm-up and before the second-long repetition below:
        # a GPU that has just run GEMMs for a second is clocked down by the power cap, and a baseline
        # timed only then would look slower than it is
        for _ in range(max(args.warmup, 3)):
            baseline_step()
        baseline_ms, _ = timed(baseline_step, args.steps)
        region_s = max(ms_per_step * args.steps / 1e3, 1e-3)
        for _ in range(min(40, max(1, int(1.0 / region_s)))):
            timed(step, args.steps)
    symm_mem.check_status(dev)

    # ---- end to end: H2D of the step's input, public API, D2H of a checksum ----
    def e2e_step():
        a_shard.copy_(a_host, non_blocking=True)
        smr.all_gather_matmul(a_shard, b, a_out, c_out)
        checksum_host.copy_(c_out[:, :8].float().sum().reshape(1), non_blocking=True)
        torch.cuda.current_stream().synchronize()

    for _ in range(3):
        e2e_step()
    e2e_ms, _ = timed(e2e_step, args.steps)
    symm_mem.check_status(dev)

    # ---- the same, fed the way a serving loop would feed it: two shard buffers, the copy of step i + 1
    #      on a copy stream while the kernel of step i runs; every step still copies its input from pinned
    #      memory and reads its checksum back.  One event pair around all K steps; no L2 flush inside
    #      (a step reads the gathered A and B, 314 MB, more than the L2 holds). ----
    copy_stream = torch.cuda.Stream(dev)
    main = torch.cuda.current_stream()
    shards = [torch.empty_like(a_shard) for _ in range(2)]      # push mode reads the shard locally only
    ready = [torch.cuda.Event() for _ in range(2)]
    consumed = [torch.cuda.Event() for _ in range(2)]

    def feed(j):
        copy_stream.wait_event(consumed[j])
        with torch.cuda.stream(copy_stream):
            shards[j].copy_(a_host, non_blocking=True)
            ready[j].record(copy_stream)

    def pipelined(steps):
        begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        for ev in consumed:
            ev.record(main)
        sync_all()
        begin.record(main)
        feed(0)
        for i in range(steps):
            j = i % 2
            if i + 1 < steps:
                feed(1 - j)
            main.wait_event(ready[j])
            smr.all_gather_matmul(shards[j], b, a_out, c_out)
            consumed[j].record(main)
            checksum_host.copy_(c_out[:, :8].float().sum().reshape(1), non_blocking=True)
            main.synchronize()                                   # the host has this step's result
        end.record(main)
        sync_all()
        return max_over_ranks(begin.elapsed_time(end) / steps, dev)

    pipelined(3)
    pipelined_ms = pipelined(args.steps)
    symm_mem.check_status(dev)

    per_gpu_tflops = flops / (ms_per_step * 1e-3) / 1e12
    e2e_tflops = flops / (e2e_ms * 1e-3) / 1e12 * world
    out = {
        "metric": "all_gather_matmul_tflops",
        "value": round(per_gpu_tflops * world, 2),
        "unit": "TFLOPS (aggregate over GPUs)",
        "n_gpus": world,
        "steps": args.steps,
        "warmup": max(args.warmup, 3),
        "ms_per_step": round(ms_per_step, 5),
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": round(per_gpu_tflops / PUBLISHED_TFLOPS_PER_GPU, 4),
        "dtype": "bf16",
        "data": "synthetic N(0,0.02), seeded 42+rank; random-init B",
        "config": {
            "model": "Llama-3-70B MLP up-proj, TP shard N=3584 K=8192",
            "global_batch": M_TOTAL, "seq_len": None,
            "parallelism": f"tp{world}",
            "M": M_TOTAL, "N_per_rank": N_PER_RANK, "K": K_DIM, "a_shard_rows": rows,
            "l2": "256 MB buffer overwritten before every timed step",
            "baseline": f"published fused {PUBLISHED_FUSED_US_H100} us on 8xH100 = "
                        f"{PUBLISHED_TFLOPS_PER_GPU:.1f} TFLOPS per GPU; vs_baseline is per-GPU",
        },
        "e2e": {"value": round(flops / (pipelined_ms * 1e-3) / 1e12 * world, 2),
                "unit": "TFLOPS (aggregate over GPUs)", "ms_per_step": round(pipelined_ms, 5),
                "h2d_bytes_per_step": a_host.numel() * 2, "d2h_bytes_per_step": 4,
                "how": "public API; every step copies its A shard from pinned host memory (on a copy stream, under "
                       "the previous step's kernel: two shard buffers) and reads a checksum of C back to the host",
                "l2": "no flush between steps: a step reads 314 MB (gathered A and B)"},
        "e2e_serial": {"value": round(e2e_tflops, 2), "unit": "TFLOPS (aggregate over GPUs)",
                       "ms_per_step": round(e2e_ms, 5),
                       "h2d_bytes_per_step": a_host.numel() * 2, "d2h_bytes_per_step": 4,
                       "how": "copy, kernel and read-back one after the other on one stream, L2 flushed per step"},
        "same_box_baseline": {
            "what": "NCCL all_gather_into_tensor + cuBLAS torch.matmul" if distributed else
                    "cuBLAS torch.matmul alone (nothing to gather at one GPU)",
            "ms_per_step": round(baseline_ms, 5), "speedup": round(baseline_ms / ms_per_step, 4)},
        # the fused kernel, and the one that adds up the K parts of a thinly filled last wave of tiles
        "gpu_launches": args.steps * C.gemm_kernels(M_TOTAL, N_PER_RANK, K_DIM, 2, sms, distributed),
        "clocks": clocks.summary(),
        "wall_s_timed_region": round(wall, 4),
    }
    if distributed and not args.no_extras:
        # the other half of the metric; a section that fails is reported, not fatal to the headline
        for key, section in (("all_reduce", all_reduce_section), ("gemv_all_reduce", gemv_section)):
            try:
                out[key] = section(world, rank, dev)
            except Exception as e:  # noqa: BLE001
                out[key] = {"failed": f"{type(e).__name__}: {e}"}
                break          # the ranks may no longer be in step: skip what follows
    if rank == 0:
        print(json.dumps(out))
    symm_mem.shutdown()
    if distributed:
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
