"""DistributedDataParallel integration.

Stock ``DistributedDataParallel`` works over the backend unchanged (it issues
one SUM allreduce per gradient bucket after dividing the bucket by the world
size in a separate elementwise pass).  The hooks here remove that extra pass:

* :func:`fused_avg_hook` -- the bucket is reduced by ONE kernel that also
  applies the 1/world scale (and, with ``MCCL_WIRE_DTYPE``, the fp32<->bf16
  wire cast) in its epilogue.
* :func:`topk_hook` -- fused top-k compressed allreduce with error feedback
  (select -> sparse exchange over NVLink -> deterministic scatter-add); the
  residual lives in a per-bucket fp32 buffer keyed by the bucket index.

Both return futures that are ordered on the communication stream, so no host
synchronisation happens between backward and the optimizer step.
"""
import os
import weakref
from typing import Dict, Optional

import torch
import torch.distributed as dist
from torch.nn.parallel import DistributedDataParallel

from ..ops.linear import Linear


# layers whose products are torch's for the sake of a compressed wrapper: layer -> token of that wrapper
_torch_product_layers = weakref.WeakKeyDictionary()


def _own_products(module, owner=None) -> None:
    """Undoes :func:`_torch_products` in ``module``: all of it, or what the wrapper ``owner`` has done."""
    for m in module.modules():
        token = _torch_product_layers.get(m)
        if token is not None and (owner is None or token is owner):
            m.stock = False
            del _torch_product_layers[m]


def _torch_products(ddp, module) -> None:
    """Compressed training sends what the largest fp32 gradients are, which the last bit of a product can decide: while such
    a wrapper lives, the module's layers keep torch's products.  Layers whose ``stock`` the program has set stay as they are."""
    token = object()
    for m in module.modules():
        if isinstance(m, Linear) and not m.stock:
            m.stock = True
            _torch_product_layers[m] = token
    module = weakref.ref(module)

    def release():
        if module() is not None:
            _own_products(module(), token)

    weakref.finalize(ddp, release).atexit = False


def _backend_for(process_group, device):
    pg = process_group if process_group is not None else dist.distributed_c10d._get_default_group()
    return pg._get_backend(device)


def fused_avg_hook(process_group, bucket: dist.GradBucket) -> torch.futures.Future[torch.Tensor]:
    """DDP comm hook: ``bucket = sum_over_ranks(bucket) / world`` in one fused kernel."""
    buf = bucket.buffer()
    backend = _backend_for(process_group, buf.device)
    world = backend.size()
    work = backend.allreduce_scaled(buf, 1.0 / world)
    return work.get_future().then(lambda f: f.value()[0])


class TopKState:
    """Per-model state of :func:`topk_hook`: ratio and one fp32 residual per bucket."""

    def __init__(self, process_group=None, ratio: Optional[float] = None, warmup_dense_steps: int = 0):
        self.process_group = process_group
        self.ratio = float(ratio if ratio is not None else os.environ.get("MCCL_TOPK_RATIO", "0.01"))
        if not (0.0 < self.ratio <= 1.0):
            raise ValueError("ratio must be in (0, 1]")
        self.residuals: Dict[int, torch.Tensor] = {}
        self.warmup_dense_steps = warmup_dense_steps
        self.calls = 0

    def residual_for(self, bucket: dist.GradBucket) -> torch.Tensor:
        buf = bucket.buffer()
        idx = bucket.index()
        r = self.residuals.get(idx)
        if r is None or r.numel() != buf.numel() or r.device != buf.device:
            r = torch.zeros(buf.numel(), dtype=torch.float32, device=buf.device)
            self.residuals[idx] = r
        return r

    def reset(self) -> None:
        """Drops all residuals (they also restart at zero after a checkpoint resume)."""
        self.residuals.clear()


def topk_hook(state: TopKState, bucket: dist.GradBucket) -> torch.futures.Future[torch.Tensor]:
    """DDP comm hook: top-k compressed gradient averaging with error feedback."""
    buf = bucket.buffer()
    backend = _backend_for(state.process_group, buf.device)
    world = backend.size()
    if bucket.index() == 0:
        state.calls += 1
    if state.calls <= state.warmup_dense_steps:
        work = backend.allreduce_scaled(buf, 1.0 / world)
    else:
        work = backend.allreduce_topk(buf, state.residual_for(bucket), state.ratio, 1.0 / world)
    return work.get_future().then(lambda f: f.value()[0])


class OptimizerInBackward:
    """State of :func:`optimizer_in_backward_hook`: the fused optimizer and the process group."""

    def __init__(self, optimizer, process_group=None):
        self.optimizer = optimizer
        self.process_group = process_group
        self.backend = None   # resolved on first use
        self.scale = 1.0


def optimizer_in_backward_hook(state: OptimizerInBackward, bucket: dist.GradBucket) -> torch.futures.Future[torch.Tensor]:
    """DDP comm hook: fused-average allreduce, then the bucket's AdamW update, both off the main stream.

    One native call per bucket enqueues the allreduce kernel and, right behind it on the same
    communication stream, the AdamW kernel over the bucket's parameters; the returned future
    covers both.  The update therefore runs while later buckets are still being reduced and
    backward is still computing.  ``optimizer.step()`` afterwards only refreshes the step
    counters (and covers parameters that were not updated here, normally none).
    """
    buf = bucket.buffer()
    backend = state.backend
    if backend is None:
        backend = state.backend = _backend_for(state.process_group, buf.device)
        state.scale = 1.0 / backend.size()
    opt = state.optimizer
    if bucket.index() == 0:
        opt.begin_step_in_backward()
    plans = opt.bucket_plans(bucket.index(), bucket.parameters())
    grads = bucket.gradients()
    specs = []
    for plan, group, own, pos in plans:
        b1, b2 = group["betas"]
        specs.append((plan, [grads[i] for i in pos], group["lr"], b1, b2, group["eps"], group["weight_decay"]))
        opt.mark_bucket_stepped(own)
    work = backend.allreduce_adamw(buf, state.scale, specs, opt._bw_step)
    return work.get_future().then(_first_tensor)


def _first_tensor(fut):
    return fut.value()[0]


def _install_native_bucket_hook(ddp, optimizer, process_group) -> None:
    """Registers the C++ allreduce+AdamW hook on DDP's reducer (no Python per bucket).

    The optimizer's state is created up front and handed to the hook; a forward pre-hook pushes the
    current hyper-parameters and step number before every iteration.
    """
    from .. import require_native

    native = require_native()
    device = next(ddp.module.parameters()).device
    backend = _backend_for(process_group, device)
    state = native.BucketOptimizerState(backend, 1.0 / backend.size())
    optimizer.attach_native_hook(state)
    native._register_bucket_optimizer_hook(ddp.reducer, state)
    ddp._mccl_native_hook_state = state
    ddp.register_forward_pre_hook(lambda _m, _inp: optimizer.sync_native_hook())


def nvls_tensor_pool(nbytes: int, process_group=None, device=None):
    """A ``torch.cuda.MemPool`` of ``nbytes`` of multicast-bound device memory, or None.

    Tensors allocated inside ``with torch.cuda.use_mem_pool(pool):`` are reduced IN PLACE by the
    NVSwitch when they are passed to ``all_reduce`` (SUM / AVG of fp32, fp16, bf16; byte length a
    multiple of 16): no staging copies.  Collective: every rank calls it with the same size, and
    every rank must then allocate the same sizes in the same order (a tensor has to sit at the same
    offset on all ranks; the backend checks this the first time it sees a tensor and falls back to
    the staged kernels otherwise).  One pool per device and process.  Returns None when the group
    has no NVLS (``MCCL_NVLS=0``, no NVSwitch multicast, world size 1).
    """
    from .. import require_native

    if os.environ.get("MCCL_NVLS", "auto") in ("0", "off") or not dist.is_initialized():
        return None
    if device is None:
        device = torch.device("cuda", torch.cuda.current_device())
    device = torch.device(device)
    backend = _backend_for(process_group, device)
    if backend.size() < 2 or not hasattr(backend, "create_nvls_user_pool"):
        return None
    want = (int(nbytes) + (1 << 21) - 1) // (1 << 21) * (1 << 21)
    if not backend.create_nvls_user_pool(want, device.index):
        return None
    native = require_native()
    alloc = torch.cuda.memory.CUDAPluggableAllocator(native.__file__, "mccl_nvls_pool_alloc", "mccl_nvls_pool_free")
    pool = torch.cuda.MemPool(alloc.allocator())
    pool._mccl_allocator = alloc  # keep the ctypes handles alive as long as the pool
    return pool


def _nvls_bucket_pool(module: torch.nn.Module, process_group):
    """A ``torch.cuda.MemPool`` whose memory is bound to the group's NVLink multicast object, or None.

    Gradient buckets allocated from it are reduced IN PLACE by the NVSwitch (``multimem.ld_reduce`` /
    ``multimem.st`` straight on the bucket): no staging copies, (1 + 1/world) x bytes per link
    direction and only world-th of the bucket handled by each GPU's SMs.  Collective: every rank must
    call it (``wrap_ddp`` does).  Returns None when NVLS is unavailable, switched off
    (``MCCL_NVLS=0`` / ``MCCL_NVLS_BUCKETS=0``) or the world size is 1.
    """
    if os.environ.get("MCCL_NVLS_BUCKETS", "1") == "0" or os.environ.get("MCCL_NVLS", "auto") in ("0", "off"):
        return None
    params = [p for p in module.parameters() if p.requires_grad]
    if not params or not params[0].is_cuda:
        return None
    device = params[0].device
    backend = _backend_for(process_group, device)
    # With two ranks the in-switch reduction has no traffic advantage over the one-shot exchange
    # (measured: 72.1 k vs 73.9 k samples/s on the 94 M MLP), so the pool is used from 4 ranks on.
    min_world = int(os.environ.get("MCCL_NVLS_BUCKETS_MIN_WORLD", "4"))
    if backend.size() < max(2, min_world) or not hasattr(backend, "create_nvls_user_pool"):
        return None
    need = sum(p.numel() * p.element_size() for p in params)
    # buckets are rebuilt once after the first backward, and a process may wrap a model more than once
    # before the first wrapper's memory is back: room for four generations plus slack
    want = int(os.environ.get("MCCL_NVLS_POOL_BYTES", "0")) or (4 * need + (256 << 20))
    return nvls_tensor_pool(want, process_group, device)


def wrap_ddp(module: torch.nn.Module, *, device_ids=None, bucket_cap_mb: Optional[int] = None,
             compression: Optional[str] = None, fused_average: bool = True, process_group=None,
             optimizer_in_backward=None, nvls_buckets: Optional[bool] = None,
             **ddp_kwargs) -> DistributedDataParallel:
    """``DistributedDataParallel`` with the backend's fused hooks installed.

    ``compression`` (default: ``MCCL_COMPRESSION``) selects ``"topk"`` for the
    compressed hook; otherwise, on CUDA, the fused-average hook replaces DDP's
    separate divide pass.  ``bucket_cap_mb`` defaults to ``DDP_BUCKET_MB`` or 25.
    ``optimizer_in_backward`` takes a :class:`mccl_b200.optim.FusedAdamW` built over the
    module's parameters: each bucket is then updated right behind its allreduce (see
    :func:`optimizer_in_backward_hook`); keep calling ``optimizer.step()`` once per iteration.
    ``nvls_buckets`` (default: on where the group has NVLS and the gradients are reduced densely)
    places DDP's gradient buckets in multicast-bound memory so that their allreduce runs in place
    inside the NVSwitch (see :func:`_nvls_bucket_pool`).
    """
    if bucket_cap_mb is None:
        bucket_cap_mb = int(os.environ.get("DDP_BUCKET_MB", "25"))
    ddp_kwargs.setdefault("gradient_as_bucket_view", True)
    on_cuda = next(module.parameters()).is_cuda
    mode = compression if compression is not None else os.environ.get("MCCL_COMPRESSION", "none")
    _own_products(module)
    pool = None
    if on_cuda and mode != "topk" and nvls_buckets is not False and dist.is_initialized():
        pool = _nvls_bucket_pool(module, process_group)
    if pool is not None:
        with torch.cuda.use_mem_pool(pool):
            ddp = DistributedDataParallel(module, device_ids=device_ids, bucket_cap_mb=bucket_cap_mb,
                                          process_group=process_group, **ddp_kwargs)
        ddp._mccl_nvls_pool = pool
        state = {"rebuilt": False}

        def _rebuild_in_pool(_m, _inp):
            # DDP re-buckets once, at the start of the second iteration: make the new buckets come
            # from the same memory (its own call right after this one then finds nothing to do)
            if not state["rebuilt"] and torch.is_grad_enabled():
                rebuild = getattr(ddp.reducer, "_rebuild_buckets", None)
                if rebuild is None:  # a torch without this entry point: DDP's own rebuild then leaves the
                    state["rebuilt"] = True  # pool, and the backend falls back to its staged kernels
                    return
                with torch.cuda.use_mem_pool(pool):
                    if rebuild():
                        state["rebuilt"] = True

        ddp.register_forward_pre_hook(_rebuild_in_pool)
    else:
        ddp = DistributedDataParallel(module, device_ids=device_ids, bucket_cap_mb=bucket_cap_mb,
                                      process_group=process_group, **ddp_kwargs)
    if on_cuda and optimizer_in_backward is not None and mode != "topk":
        if os.environ.get("MCCL_PYTHON_BUCKET_HOOK", "0") == "1":
            ddp._mccl_oib_state = OptimizerInBackward(optimizer_in_backward, process_group)
            ddp.register_comm_hook(ddp._mccl_oib_state, optimizer_in_backward_hook)
        else:
            _install_native_bucket_hook(ddp, optimizer_in_backward, process_group)
    elif on_cuda and mode == "topk":
        _torch_products(ddp, module)
        ddp._mccl_topk_state = TopKState(process_group)
        ddp.register_comm_hook(ddp._mccl_topk_state, topk_hook)
    elif on_cuda and fused_average:
        ddp.register_comm_hook(process_group, fused_avg_hook)
    return ddp
