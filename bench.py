#!/usr/bin/env python
"""Headline benchmark: DDP training throughput (samples/s) of the ~94 M parameter fp32 MLP.

    python bench.py --gpus 1 --steps 30 --warmup 5
    python -m torch.distributed.run --nnodes=1 --nproc-per-node 8 --master-addr 127.0.0.1 \
        --master-port 29511 bench.py --gpus 8 --steps 30 --warmup 5

Config (fixed): Linear(2048,3072)-GELU, 9x[Linear(3072,3072)-GELU], Linear(3072,1000); fp32;
global batch 256 split over the ranks (strong scaling); AdamW lr 1e-3; DDP bucket 25 MB;
synthetic N(0,1) inputs and uniform labels; random-init weights.

Two timed regions, both bracketed by barrier + synchronize and timed on the device with
CUDA events (max over ranks):
  value  K full training steps (forward, backward with bucketed gradient allreduce,
         optimizer step) on device-resident inputs;
  e2e    K steps through the same public API where every step also copies its inputs from
         pinned host memory to the device and reads the loss back to the host
         (``mccl_b200.utils.data``: the copy of batch i+1 is enqueued behind step i on a side
         stream, and step i-1's loss is read while step i is being launched; the last loss is
         read before the clock stops; the same loop drives every arm).
``--impl mccl`` (default) is this framework: backend "mccl", DDP gradient buckets in
multicast-bound memory reduced in place by the NVSwitch (4 ranks and more), the native
allreduce + AdamW bucket hook (more than one rank), fused AdamW kernel.  After the headline arm
the same process measures two comparison arms with the same steps and warm-up: this backend with
torch's own fused AdamW (``no_fused_optim``: isolates the communication path) and torch's stock
NCCL backend + stock DDP + torch AdamW (``nccl_value``, ``nccl_e2e``, ``vs_nccl``,
``vs_nccl_e2e``); ``--no-compare`` skips them.  ``--impl nccl`` runs the NCCL arm alone.  ``--impl reference`` would run the unmodified reference package,
which builds only on macOS/Apple Silicon, so it prints its `unavailable` line.
"""
from __future__ import annotations

import argparse
import json
import os
import sys
import threading
import time

REFERENCE_SAMPLES_PER_S = {1: 78.3, 2: 134.2}  # reference's published numbers (Apple GPUs)
GLOBAL_BATCH = 256
IN_FEATURES, CLASSES = 2048, 1000


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=100)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="mccl", choices=["mccl", "nccl", "reference"])
    ap.add_argument("--bucket-mb", type=int, default=25)
    ap.add_argument("--no-fused-hook", action="store_true", help="stock DDP divide + SUM allreduce")
    ap.add_argument("--no-fused-optim", action="store_true", help="torch.optim.AdamW instead of the fused kernel")
    ap.add_argument("--no-compare", action="store_true",
                    help="skip the in-process comparison arms (mccl + torch AdamW, and torch's NCCL backend)")
    ap.add_argument("--optim-in-backward", default="auto", choices=["auto", "on", "off"],
                    help="AdamW per bucket right behind its allreduce (native DDP hook) instead of one step after "
                         "backward.  auto = on when there is more than one rank (measured: +2.7 %% at 2 GPUs, "
                         "+8 to +14 %% at 4 GPUs together with the in-switch bucket reduction; -1.8 %% at 1 GPU, "
                         "where there is no communication to hide the update behind)")
    return ap.parse_args()


class ClockSampler(threading.Thread):
    """Samples SM clocks and throttle reasons of one GPU through NVML while a region is timed."""

    def __init__(self, index: int, period_s: float = 0.02):
        super().__init__(daemon=True)
        self.index, self.period = index, period_s
        self.samples, self.reasons, self.max_mhz = [], set(), None
        self._stop_evt = threading.Event()
        self.ok = False
        try:
            import pynvml
            pynvml.nvmlInit()
            self.nv = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM)
            self.ok = True
        except Exception:
            self.nv = None

    def run(self):
        if not self.ok:
            return
        nv = self.nv
        names = {
            nv.nvmlClocksThrottleReasonHwSlowdown: "hw_slowdown",
            nv.nvmlClocksThrottleReasonHwThermalSlowdown: "hw_thermal_slowdown",
            nv.nvmlClocksThrottleReasonSwThermalSlowdown: "sw_thermal_slowdown",
            nv.nvmlClocksThrottleReasonSwPowerCap: "sw_power_cap",
        }
        while not self._stop_evt.is_set():
            try:
                self.samples.append(nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM))
                mask = nv.nvmlDeviceGetCurrentClocksThrottleReasons(self.h)
                for bit, name in names.items():
                    if mask & bit:
                        self.reasons.add(name)
            except Exception:
                pass
            time.sleep(self.period)

    def stop(self):
        self._stop_evt.set()
        if self.is_alive():
            self.join(timeout=2)
        s = sorted(self.samples)
        return {"sm_mhz": (s[len(s) // 2] if s else None), "sm_max_mhz": self.max_mhz,
                "reasons": sorted(self.reasons), "samples": len(s)}


def main():
    args = parse_args()
    if args.impl == "reference":
        print(json.dumps({
            "impl": "reference",
            "unavailable": "reference builds only on macOS/Apple Silicon (setup.py raises 'MCCL can only be "
                           "built on macOS' on Linux); its Metal/MPS path cannot run on this box"}))
        return 0

    import torch
    import torch.distributed as dist

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.gpus != world:
        if world == 1 and args.gpus > 1:
            sys.exit("bench.py --gpus N>1 must be launched with torch.distributed.run (one rank per GPU)")
        args.gpus = world
    os.environ.setdefault("MASTER_ADDR", "127.0.0.1")
    os.environ.setdefault("MASTER_PORT", "29533")
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)

    if args.impl == "mccl":
        import mccl_b200 as mccl
        native = mccl.require_native()
        dist.init_process_group("mccl", rank=rank, world_size=world, device_id=dev)
    else:
        native = None
        dist.init_process_group("nccl", rank=rank, world_size=world, device_id=dev)

    from mccl_b200.models import MLP94M, num_parameters
    from mccl_b200.utils.data import AsyncScalarReader, DevicePrefetcher

    local_batch = GLOBAL_BATCH // world
    assert local_batch * world == GLOBAL_BATCH, "global batch 256 must divide by the world size"
    g = torch.Generator().manual_seed(1234 + rank)
    n_host_batches = 8
    host_x = [torch.randn(local_batch, IN_FEATURES, generator=g).pin_memory() for _ in range(n_host_batches)]
    host_y = [torch.randint(0, CLASSES, (local_batch,), generator=g).pin_memory() for _ in range(n_host_batches)]
    dev_x = [t.to(dev) for t in host_x]
    dev_y = [t.to(dev) for t in host_y]
    h2d_bytes = host_x[0].nbytes + host_y[0].nbytes
    d2h_bytes = 4
    loss_fn = torch.nn.CrossEntropyLoss()
    warmup = max(args.warmup, 3)

    def run_arm(kind, fused_optim, group, torch_products=False):
        """One complete measurement (warm-up, device-timed region, end-to-end region) of one arm.

        kind "mccl": this backend + fused-average hook (+ fused AdamW when `fused_optim`);
        kind "nccl": torch's NCCL backend + stock DDP + torch.optim.AdamW(fused=True).
        `torch_products`: the model's layers use torch's fp32 matrix products (see mccl_b200/ops/linear.py).
        `group` is the process group the arm trains on (None: the default group).
        """
        torch.manual_seed(42)
        model = MLP94M().to(dev)
        for layer in model.net[::2]:
            layer.stock = torch_products
        n_params = num_parameters(model)
        in_bw = False
        if kind == "mccl":
            from mccl_b200.parallel import wrap_ddp
            from mccl_b200.optim import FusedAdamW
            opt = (FusedAdamW(model.parameters(), lr=1e-3) if fused_optim
                   else torch.optim.AdamW(model.parameters(), lr=1e-3, fused=True))
            want_bw = args.optim_in_backward == "on" or (args.optim_in_backward == "auto" and world > 1)
            in_bw = want_bw and fused_optim and not args.no_fused_hook
            ddp = wrap_ddp(model, device_ids=[local_rank], bucket_cap_mb=args.bucket_mb,
                           fused_average=not args.no_fused_hook, compression="none", process_group=group,
                           optimizer_in_backward=opt if in_bw else None)
        else:
            from torch.nn.parallel import DistributedDataParallel
            ddp = DistributedDataParallel(model, device_ids=[local_rank], bucket_cap_mb=args.bucket_mb,
                                          gradient_as_bucket_view=True, process_group=group)
            opt = torch.optim.AdamW(ddp.parameters(), lr=1e-3, fused=True)

        def train_step(x, y):
            opt.zero_grad()  # set_to_none: DDP re-points grads at its bucket views, no memset pass
            loss = loss_fn(ddp(x), y)
            loss.backward()
            opt.step()
            return loss

        # What a program sets up once: the copy stream with its device memory, and the pinned slots of the loss.  (Allocated
        # inside the clock they took 1 ms of a 20-step region, and whatever else the driver was busy with.)
        copy_stream = torch.cuda.Stream(dev)
        losses = AsyncScalarReader(dev)

        def e2e_steps(n):
            # every step: its inputs come from pinned host memory (copy of batch i+1 behind step i) and
            # its loss is read on the host (step i-1's while step i is being launched; the last one
            # before the clock stops)
            feed = DevicePrefetcher(((host_x[i % n_host_batches], host_y[i % n_host_batches]) for i in range(n)), dev,
                                    stream=copy_stream)
            for i in range(n):
                x, y = feed.next()
                losses.push(train_step(x, y))
                if i > 0:
                    losses.pop()
            return losses.pop()

        def timed(region_steps, e2e):
            torch.cuda.synchronize()
            dist.barrier(group=group)
            torch.cuda.synchronize()
            sampler = ClockSampler(local_rank)
            sampler.start()
            launches0 = native._kernel_launches() if native else 0
            start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0 = time.perf_counter()
            start.record()
            last = None
            if e2e:
                last = e2e_steps(region_steps)
            else:
                for i in range(region_steps):
                    last = train_step(dev_x[i % n_host_batches], dev_y[i % n_host_batches])
            end.record()
            torch.cuda.synchronize()
            wall_ms = (time.perf_counter() - t0) * 1e3
            dist.barrier(group=group)
            torch.cuda.synchronize()
            clocks = sampler.stop()
            launches = (native._kernel_launches() - launches0) if native else 0
            dev_ms = start.elapsed_time(end)
            # e2e is a host-visible quantity: take the larger of device and wall time
            ms = max(dev_ms, wall_ms) if e2e else dev_ms
            t = torch.tensor([ms], dtype=torch.float64, device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX, group=group)
            if not e2e and not isinstance(last, float):
                last = float(last.item())
            return float(t.item()), clocks, launches, last

        pooled = getattr(ddp, "_mccl_nvls_pool", None) is not None
        for i in range(warmup):
            train_step(dev_x[i % n_host_batches], dev_y[i % n_host_batches])
        ms_total, clocks, launches, _ = timed(args.steps, e2e=False)
        e2e_steps(4)
        ms_e2e, clocks_e2e, _, loss_b = timed(args.steps, e2e=True)
        del ddp, opt, model
        torch.cuda.empty_cache()
        return {"ms_total": ms_total, "ms_e2e": ms_e2e, "clocks": clocks, "clocks_e2e": clocks_e2e,
                "launches": launches, "final_loss": loss_b, "n_params": n_params, "in_bw": in_bw, "pooled": pooled,
                "value": GLOBAL_BATCH / (ms_total / args.steps / 1e3),
                "e2e_value": GLOBAL_BATCH / (ms_e2e / args.steps / 1e3)}

    main_arm = run_arm(args.impl, not args.no_fused_optim, None, torch_products=args.impl == "nccl")
    ms_total, ms_e2e = main_arm["ms_total"], main_arm["ms_e2e"]
    clocks, clocks_e2e, launches, loss_b = main_arm["clocks"], main_arm["clocks_e2e"], main_arm["launches"], main_arm["final_loss"]
    n_params, in_bw = main_arm["n_params"], main_arm["in_bw"]

    # Comparison arms in the same process, on the same GPUs, with the same steps and warm-up:
    # (a) this backend with torch's own fused AdamW, which isolates the communication path from the
    # optimizer kernel, (b) torch's stock NCCL backend + stock DDP + torch AdamW under the same model, and (c) the same
    # with torch's own matrix products in the model's layers.
    extra = {}
    if args.impl == "mccl" and not args.no_compare:
        if not args.no_fused_optim:
            arm = run_arm("mccl", False, None)
            extra["no_fused_optim"] = {"value": round(arm["value"], 2), "e2e": round(arm["e2e_value"], 2),
                                       "ms_per_step": round(arm["ms_total"] / args.steps, 4), "clocks": arm["clocks"]}
        try:
            nccl_group = dist.new_group(backend="nccl")
            # the backend's share of the difference: the same layers on either side
            same = run_arm("nccl", False, nccl_group)
            extra["nccl_same_layers"] = {"value": round(same["value"], 2), "e2e": round(same["e2e_value"], 2),
                                         "ms_per_step": round(same["ms_total"] / args.steps, 4), "clocks": same["clocks"]}
            extra["vs_nccl_same_layers"] = round(main_arm["value"] / same["value"], 4)
            # and torch alone, its fp32 products included
            arm = run_arm("nccl", False, nccl_group, torch_products=True)
            extra["nccl_value"] = round(arm["value"], 2)
            extra["nccl_e2e"] = round(arm["e2e_value"], 2)
            extra["nccl_ms_per_step"] = round(arm["ms_total"] / args.steps, 4)
            extra["nccl_clocks"] = arm["clocks"]
            extra["vs_nccl"] = round(main_arm["value"] / arm["value"], 4)
            extra["vs_nccl_e2e"] = round(main_arm["e2e_value"] / arm["e2e_value"], 4)
            if "no_fused_optim" in extra:
                extra["no_fused_optim"]["vs_nccl"] = round(extra["no_fused_optim"]["value"] / arm["value"], 4)
                extra["no_fused_optim"]["vs_nccl_e2e"] = round(extra["no_fused_optim"]["e2e"] / arm["e2e_value"], 4)
        except Exception as exc:  # the comparison must never take the headline down with it
            extra["nccl_error"] = f"{type(exc).__name__}: {exc}"[:300]

    ms_per_step = ms_total / args.steps
    value = GLOBAL_BATCH / (ms_per_step / 1e3)
    e2e_value = GLOBAL_BATCH / ((ms_e2e / args.steps) / 1e3)
    base = REFERENCE_SAMPLES_PER_S.get(world)
    plane = "n/a"
    if args.impl == "mccl":
        import mccl_b200 as mccl
        plane = mccl.get_backend(device=dev).data_plane()
    out = {
        "metric": "ddp_samples_per_sec",
        "value": round(value, 2),
        "unit": "samples/s",
        "n_gpus": world,
        "steps": args.steps,
        "warmup": warmup,
        "ms_per_step": round(ms_per_step, 4),
        "higher_is_better": True,
        "scaling": "strong",
        "vs_baseline": (round(value / base, 2) if base else None),
        "dtype": "fp32",
        "data": "synthetic N(0,1) inputs, uniform labels, random-init weights",
        "impl": args.impl,
        "config": {
            "model": f"MLP-94M fp32 ({n_params} params): Linear(2048,3072)-GELU, 9x[Linear(3072,3072)-GELU], Linear(3072,1000)",
            "global_batch": GLOBAL_BATCH,
            "seq_len": None,
            "parallelism": f"dp{world}",
            "optimizer": "AdamW lr=1e-3",
            "products": ("fp32 operands, results and sums; each product as six bf16 products on the tensor cores (sums no further "
                         "from 64 bits than an fp32 kernel's)" if native and native._linear_pays("forward", local_batch, 3072, 3072)
                         else "torch fp32"),
            "ddp_bucket_mb": args.bucket_mb,
            "l2": "no flush: params+grads+AdamW state are 1.5 GB per step, far above the 126 MB L2",
            "data_plane": plane,
            "fused_avg_hook": args.impl == "mccl" and not args.no_fused_hook,
            "fused_adamw": args.impl == "mccl" and not args.no_fused_optim,
            "optimizer_in_backward": args.impl == "mccl" and in_bw,
            "nvls_in_place_buckets": args.impl == "mccl" and main_arm["pooled"],
        },
        "clocks": clocks,
        "e2e": {"value": round(e2e_value, 2), "unit": "samples/s", "ms_per_step": round(ms_e2e / args.steps, 4),
                "h2d_bytes_per_step": h2d_bytes, "d2h_bytes_per_step": d2h_bytes, "clocks": clocks_e2e},
        "gpu_launches": launches,
        "final_loss": loss_b,
    }
    out.update(extra)
    if rank == 0:
        print(json.dumps(out), flush=True)
    dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
