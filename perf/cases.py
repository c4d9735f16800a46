"""Performance cases of the framework on one GPU: what is timed, on which sizes, and how close results must stay.

Five kinds of work, all through the entry points a program uses:

``stft`` / ``istft``  ``mccl_b200.transforms``: forward alone (inference) or forward and backward (training).
``adamw``             ``FusedAdamW.step()`` over the parameters of an MLP of the benchmark's family.
``topk``              the backend's ``allreduce_topk``: what the compressed DDP hook calls for each gradient bucket.
``train``             one DDP training step (``wrap_ddp`` + ``FusedAdamW``) of an MLP of the benchmark's family.
``collective``        the collective kernels with every rank of the group on this one GPU (``EmuGroup``), the form in
                      which a single device runs them; sizes and algorithm follow what the backend picks itself.

A case is a dict of plain values; :func:`prepare` turns it into what a program holds before the call, :func:`run`
makes one pass and returns everything that pass computes.
"""
from __future__ import annotations

import math

import torch
import torch.distributed as dist
import torch.nn.functional as F

import mccl_b200
from mccl_b200.models.mlp import MLP94M
from mccl_b200.optim import FusedAdamW
from mccl_b200.parallel import wrap_ddp
from mccl_b200.transforms import istft, stft

_DTYPES = {"float32": torch.float32, "bfloat16": torch.bfloat16, "float16": torch.float16}


def listed():
    return [
        # one second of 16 kHz speech, 25 ms window in a 512-point frame: the call a streaming front end makes
        {"name": "stft_clip", "kind": "stft", "batch": 1, "samples": 16000, "n_fft": 512, "hop": 128, "win": 400,
         "center": True, "normalized": False, "grad": False, "layout": "frames"},
        # two seconds of stereo-sized audio through a spectral loss: forward and backward (the guard of the test-suite)
        {"name": "stft_train_pair", "kind": "stft", "batch": 2, "samples": 48000, "n_fft": 2048, "hop": 512, "win": 2048,
         "center": True, "normalized": False, "grad": True, "layout": "frames"},
        # a training batch of long waveforms through the same loss: the largest transform of the repository's benchmark
        {"name": "stft_train_batch", "kind": "stft", "batch": 16, "samples": 1 << 20, "n_fft": 2048, "hop": 512, "win": 2048,
         "center": True, "normalized": False, "grad": True, "layout": "frames"},
        # waveform synthesis from a network's output, which is contiguous [batch, freq, frames]; odd length
        {"name": "istft_batch", "kind": "istft", "batch": 16, "samples": 240007, "n_fft": 1024, "hop": 256, "win": 1024,
         "center": True, "normalized": False, "grad": False, "layout": "bins"},
        # the optimizer of the two-layer smoke model: launch and host cost
        {"name": "adamw_tiny", "kind": "adamw", "features": 512, "hidden": 256, "depth": 0, "classes": 10},
        # the optimizer of the benchmark's MLP at full width
        {"name": "adamw_wide", "kind": "adamw", "features": 2048, "hidden": 3072, "depth": 8, "classes": 1000},
        # the first gradient bucket of a backward pass (DDP keeps it at 1 MiB), compressed to 1 %
        {"name": "topk_first_bucket", "kind": "topk", "n": 262144, "dtype": "float32", "ratio": 0.01},
        # the bucket of one 50257 x 1024 embedding: the largest bucket a model of this repository has, bf16 gradients
        {"name": "topk_embedding", "kind": "topk", "n": 50257 * 1024, "dtype": "bfloat16", "ratio": 0.01},
        # a training step with compressed gradients: several 25 MB buckets' worth of top-k behind a small backward
        {"name": "train_topk", "kind": "train", "features": 2048, "hidden": 1024, "depth": 4, "classes": 1000, "batch": 64,
         "compression": "topk", "optimizer_in_backward": False},
        # the headline workload: the 94 M parameter fp32 MLP at batch 256
        {"name": "train_mlp94m", "kind": "train", "features": 2048, "hidden": 3072, "depth": 9, "classes": 1000, "batch": 256,
         "compression": "none", "optimizer_in_backward": False},
        # a small ragged bf16 gradient over eight ranks: the latency end of the allreduce
        {"name": "allreduce_small", "kind": "collective", "op": "allreduce", "ranks": 8, "n": 10007, "dtype": "bfloat16"},
        # one 25 MB DDP bucket over four ranks: the ordinary allreduce of a training step
        {"name": "allreduce_bucket", "kind": "collective", "op": "allreduce", "ranks": 4, "n": 6553600, "dtype": "float32"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["stft", "istft", "adamw", "topk", "train", "collective"])
    if kind in ("stft", "istft"):
        n_fft = rng.choice([256, 512, 1024, 2048, 4096])
        batch = rng.choice([1, 2, 3, 5, 8, 16])
        return {"kind": kind, "batch": batch, "samples": _log_int(rng, 8000, (1 << 20) - 1), "n_fft": n_fft,
                "hop": rng.choice([n_fft // 4, n_fft // 2, n_fft // 4 + n_fft // 16]),
                "win": rng.choice([n_fft, n_fft, n_fft - n_fft // 8]),
                "center": kind == "istft" or rng.random() < 0.8, "normalized": rng.random() < 0.3,
                "grad": rng.random() < 0.6, "layout": rng.choice(["frames", "frames", "bins"])}
    if kind == "adamw":
        return {"kind": kind, "features": rng.choice([512, 1024, 2048]), "hidden": _log_int(rng, 64, 3000),
                "depth": rng.randint(0, 7), "classes": rng.randint(10, 1000)}
    if kind == "topk":
        return {"kind": kind, "n": _log_int(rng, 10000, 50257 * 1023), "dtype": rng.choice(["float32", "bfloat16"]),
                "ratio": rng.choice([0.001, 0.01, 0.1])}
    if kind == "train":
        compression = rng.choice(["none", "topk"])
        return {"kind": kind, "features": rng.choice([512, 1024, 2048]), "hidden": _log_int(rng, 256, 3000),
                "depth": rng.randint(1, 7), "classes": rng.randint(10, 1000), "batch": _log_int(rng, 8, 255),
                "compression": compression, "optimizer_in_backward": compression == "none" and rng.random() < 0.5}
    return {"kind": kind, "op": rng.choice(["allreduce", "allreduce", "reduce_scatter", "allgather", "broadcast"]),
            "ranks": rng.choice([2, 4, 8]), "n": _log_int(rng, 1000, 3000000),
            "dtype": rng.choice(["float32", "bfloat16", "float16"])}


# ---- helpers -------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _backend(device):
    """The process group of a one-process program (created once per process) and its native backend."""
    if not dist.is_initialized():
        dist.init_process_group("mccl", store=dist.HashStore(), rank=0, world_size=1)
    return mccl_b200.get_backend(device=device)


def _frames(case):
    if case["center"]:
        return 1 + case["samples"] // case["hop"]
    return 1 + (case["samples"] - case["n_fft"]) // case["hop"]


def _spectrum(case, gen, device):
    b, f, t = case["batch"], case["n_fft"] // 2 + 1, _frames(case)
    if case["layout"] == "frames":  # memory order of the framework's own spectra (and of gradients derived from them)
        return torch.randn(b, t, f, dtype=torch.complex64, generator=gen, device=device).transpose(1, 2)
    return torch.randn(b, f, t, dtype=torch.complex64, generator=gen, device=device)


def _linears(case):
    dims = [case["features"]] + [case["hidden"]] * (case["depth"] + 1) + [case["classes"]]
    return list(zip(dims[:-1], dims[1:]))


def _params(case):
    return sum(i * o + o for i, o in _linears(case))


# ---- what a program has in hand before the call -----------------------------------------------------
def prepare(case, seed):
    device = _device()
    gen = torch.Generator(device=device).manual_seed(seed)
    kind = case["kind"]
    if kind in ("stft", "istft"):
        state = {"case": case, "window": torch.hann_window(case["win"], device=device)}
        wave = 0.3 * torch.randn(case["batch"], case["samples"], generator=gen, device=device)
        spec = _spectrum(case, gen, device)
        if kind == "stft":
            state["input"] = wave.requires_grad_(case["grad"])
            state["grad_output"] = spec if case["grad"] else None
        else:
            state["input"] = spec.requires_grad_(case["grad"])
            state["grad_output"] = wave if case["grad"] else None
        return state
    if kind == "adamw":
        params = []
        for i, o in _linears(case):
            params.append(torch.nn.Parameter(torch.randn(o, i, generator=gen, device=device) / math.sqrt(i)))
            params.append(torch.nn.Parameter(torch.randn(o, generator=gen, device=device) / math.sqrt(i)))
        opt = FusedAdamW(params, lr=1e-3)
        # one step behind us, as in any iteration but the first: the moments exist and are not zero
        for p in params:
            p.grad = 1e-3 * torch.randn(p.shape, generator=gen, device=device)
        opt.step()
        for p in params:
            p.grad = 1e-3 * torch.randn(p.shape, generator=gen, device=device)
        return {"case": case, "optimizer": opt, "params": params}
    if kind == "topk":
        grad = (1e-3 * torch.randn(case["n"], generator=gen, device=device)).to(_DTYPES[case["dtype"]])
        residual = 2e-3 * torch.randn(case["n"], generator=gen, device=device)
        return {"case": case, "backend": _backend(device), "grad": grad, "residual": residual}
    if kind == "train":
        _backend(device)
        torch.manual_seed(seed)
        with torch.device(device):
            model = MLP94M(case["features"], case["hidden"], case["depth"], case["classes"])
        opt = FusedAdamW(model.parameters(), lr=1e-3)
        ddp = wrap_ddp(model, device_ids=[device.index], bucket_cap_mb=25, compression=case["compression"],
                       optimizer_in_backward=opt if case["optimizer_in_backward"] else None)
        x = torch.randn(case["batch"], case["features"], generator=gen, device=device)
        y = torch.randint(0, case["classes"], (case["batch"],), generator=gen, device=device)
        return {"case": case, "model": ddp, "optimizer": opt, "x": x, "y": y, "params": list(model.parameters())}
    # collective: the per-rank tensors and the group's arena, sized for the largest exchange (slots of every rank, twice)
    ws, n, dtype = case["ranks"], case["n"], _DTYPES[case["dtype"]]
    esz = torch.empty((), dtype=dtype).element_size()
    native = mccl_b200.require_native()
    block = n * esz
    need = {"allreduce": block * (ws if _oneshot(case) else 2), "reduce_scatter": block * ws, "allgather": block * ws,
            "broadcast": block}[case["op"]]
    group = native.EmuGroup(ws, (need + 4096 * ws + (1 << 20)) // 4096 * 4096)
    count = n * ws if case["op"] == "reduce_scatter" else n
    inputs = [torch.randn(count, generator=gen, device=device).to(dtype) for _ in range(ws)]
    outputs = None
    if case["op"] == "reduce_scatter":
        outputs = [torch.empty(n, dtype=dtype, device=device) for _ in range(ws)]
    elif case["op"] == "allgather":
        outputs = [torch.empty(n * ws, dtype=dtype, device=device) for _ in range(ws)]
    return {"case": case, "group": group, "inputs": inputs, "outputs": outputs}


def _oneshot(case):
    """The backend's measured rule: one-shot up to 32 MiB at two ranks, 4 MiB at four, 1 MiB at eight."""
    esz = torch.empty((), dtype=_DTYPES[case["dtype"]]).element_size()
    return case["n"] * esz <= {2: 32 << 20, 4: 4 << 20, 8: 1 << 20}[case["ranks"]]


# ---- one pass ---------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("stft", "istft"):
        kw = dict(n_fft=case["n_fft"], hop_length=case["hop"], win_length=case["win"], window=state["window"],
                  center=case["center"], normalized=case["normalized"])
        if kind == "stft":
            out = stft(state["input"], **kw)
        else:
            out = istft(state["input"], length=case["samples"], **kw)
        if not case["grad"]:
            return out
        (grad,) = torch.autograd.grad(out, state["input"], state["grad_output"])
        return [out.detach(), grad]
    if kind == "adamw":
        opt = state["optimizer"]
        opt.step()
        params = state["params"]
        return {"params": [p.detach() for p in params], "exp_avg": [opt.state[p]["exp_avg"] for p in params],
                "exp_avg_sq": [opt.state[p]["exp_avg_sq"] for p in params]}
    if kind == "topk":
        state["backend"].allreduce_topk(state["grad"], state["residual"], case["ratio"], 1.0).wait()
        return [state["grad"], state["residual"]]
    if kind == "train":
        opt = state["optimizer"]
        opt.zero_grad()
        loss = F.cross_entropy(state["model"](state["x"]), state["y"])
        loss.backward()
        opt.step()
        return {"loss": loss.detach(), "weights": [p.detach() for p in state["params"]],
                "grads": [p.grad for p in state["params"]]}
    group, ins, outs = state["group"], state["inputs"], state["outputs"]
    if case["op"] == "allreduce":
        if _oneshot(case):
            group.allreduce(ins, "avg", "oneshot")
        else:
            group.allreduce(ins, "avg", "twoshot", push_gather=True)
        return ins
    if case["op"] == "reduce_scatter":
        group.reduce_scatter(outs, ins, "avg")
        return outs
    if case["op"] == "allgather":
        group.allgather(outs, ins)
        return outs
    group.broadcast(ins, 0)
    return ins


# ---- what one pass cannot do without ------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("stft", "istft"):
        n_fft, frames = case["n_fft"], _frames(case)
        wave = case["batch"] * case["samples"] * 4
        spec = case["batch"] * frames * (n_fft // 2 + 1) * 8
        passes = 2 if case["grad"] else 1
        # a real FFT of n points: about 2.5 n log2 n operations
        return {"bytes": passes * (wave + spec),
                "flops": passes * case["batch"] * frames * 2.5 * n_fft * math.log2(n_fft)}
    if kind == "adamw":
        return {"bytes": 28 * _params(case), "flops": 14 * _params(case)}
    if kind == "topk":
        g = 4 if case["dtype"] == "float32" else 2
        # gradient read and written, residual read and written
        return {"bytes": case["n"] * (2 * g + 8), "flops": 2 * case["n"]}
    if kind == "train":
        weights = [i * o for i, o in _linears(case)]
        # forward, weight gradient and (but for the first layer) input gradient; p, m, v read and written, gradients written
        return {"bytes": 28 * _params(case) + 4 * case["batch"] * case["features"],
                "flops": case["batch"] * (6 * sum(weights) - 2 * weights[0])}
    esz = 4 if case["dtype"] == "float32" else 2
    ws, block = case["ranks"], case["n"] * esz
    moved = {"allreduce": 2 * ws * block, "reduce_scatter": ws * (ws + 1) * block, "allgather": ws * (ws + 1) * block,
             "broadcast": ws * block}[case["op"]]
    return {"bytes": moved, "flops": case["n"] * ws * (ws - 1) if case["op"] in ("allreduce", "reduce_scatter") else 0}


def tolerance(case):
    """About four times the distance to the same path in 64 bits, as measured over the listed and two dozen drawn cases."""
    kind = case["kind"]
    if kind in ("stft", "istft"):
        return {"rel": 6e-7, "max": 3.5e-6}
    if kind == "adamw":
        return {"rel": 3.2e-5, "max": 5.2e-5}  # the second moment: 1 - beta2 is a rounded fp32 difference (8e-6)
    if kind == "topk":
        return "exact"  # one fp32 addition per element, a selection with defined ties, one rounding to the gradient's type
    if kind == "train":
        return {"rel": 5e-5, "max": 3e-3}  # AdamW divides by the root of a second moment that is nearly zero at step one
    if case["op"] in ("allgather", "broadcast"):
        return "exact"
    # sums of up to eight values carried in fp32 (another order differs by an ulp or two), rounded once to the tensor's type
    return {"float32": {"rel": 3e-7, "max": 2e-6}, "bfloat16": {"rel": 8e-3, "max": 1.6e-2},
            "float16": {"rel": 1e-3, "max": 2e-3}}[case["dtype"]]


# ---- the same results in 64 bits, from plain torch ------------------------------------------------------
def _padded_window(case, device):
    n, win = case["n_fft"], case["win"]
    left = (n - win) // 2
    return F.pad(torch.hann_window(win, device=device).double(), (left, n - win - left))


def _overlap_add(frames, hop):
    """[..., frames, n_fft] to [..., n_fft + hop * (frames - 1)]."""
    count, n = frames.shape[-2:]
    at = (torch.arange(count, device=frames.device)[:, None] * hop + torch.arange(n, device=frames.device)).reshape(-1)
    out = frames.new_zeros(*frames.shape[:-2], n + hop * (count - 1))
    return out.index_add(-1, at, frames.flatten(-2))


def _stft64(x, case):
    n, hop = case["n_fft"], case["hop"]
    if case["center"]:
        x = F.pad(x[:, None], (n // 2, n // 2), mode="reflect")[:, 0]
    spec = torch.fft.rfft(x.unfold(-1, n, hop) * _padded_window(case, x.device))
    return (spec / math.sqrt(n) if case["normalized"] else spec).transpose(1, 2)


def _istft64(spec, case):
    n, hop, length = case["n_fft"], case["hop"], case["samples"]
    win = _padded_window(case, spec.device)
    frames = torch.fft.irfft(spec.transpose(1, 2), n=n) * win
    if case["normalized"]:
        frames = frames * math.sqrt(n)
    y = _overlap_add(frames, hop)
    env = _overlap_add((win * win).expand(spec.shape[2], n), hop)
    y = torch.where(env > 1e-11, y / env.clamp_min(1e-11), torch.zeros_like(y))
    y = y[:, n // 2:n // 2 + length]
    return F.pad(y, (0, length - y.shape[-1]))


def _adamw64(params, grads, moments, step):
    """One step of AdamW with the default betas, eps and weight decay and lr 1e-3, in place; `step` counts from 1."""
    for p, g, (m, v) in zip(params, grads, moments):
        p.mul_(1 - 1e-3 * 1e-2)
        m.mul_(0.9).add_(g, alpha=1 - 0.9)
        v.mul_(0.999).addcmul_(g, g, value=1 - 0.999)
        p.sub_(1e-3 / (1 - 0.9 ** step) * m / (v.sqrt() / math.sqrt(1 - 0.999 ** step) + 1e-8))


def exact(case, seed):
    device = _device()
    gen = torch.Generator(device=device).manual_seed(seed)
    kind = case["kind"]
    if kind in ("stft", "istft"):
        wave = (0.3 * torch.randn(case["batch"], case["samples"], generator=gen, device=device)).double()
        spec = _spectrum(case, gen, device).to(torch.complex128)
        x, other, fn = (wave, spec, _stft64) if kind == "stft" else (spec, wave, _istft64)
        if not case["grad"]:
            return fn(x, case)
        x.requires_grad_(True)
        out = fn(x, case)
        (grad,) = torch.autograd.grad(out, x, other)
        return [out.detach(), grad]
    if kind == "adamw":
        params = []
        for i, o in _linears(case):
            params.append((torch.randn(o, i, generator=gen, device=device) / math.sqrt(i)).double())
            params.append((torch.randn(o, generator=gen, device=device) / math.sqrt(i)).double())
        moments = [(torch.zeros_like(p), torch.zeros_like(p)) for p in params]
        for step in (1, 2):
            grads = [(1e-3 * torch.randn(p.shape, generator=gen, device=device)).double() for p in params]
            _adamw64(params, grads, moments, step)
        return {"params": params, "exp_avg": [m for m, _ in moments], "exp_avg_sq": [v for _, v in moments]}
    if kind == "topk" or (kind == "train" and case["compression"] == "topk"):
        return None  # which entries are sent is decided on fp32 sums: another precision sends others
    if kind == "train":
        torch.manual_seed(seed)
        with torch.device(device):
            layers = [torch.nn.Linear(i, o) for i, o in _linears(case)]
        x = torch.randn(case["batch"], case["features"], generator=gen, device=device).double()
        y = torch.randint(0, case["classes"], (case["batch"],), generator=gen, device=device)
        for n, layer in enumerate(layers):
            x = layer.double()(x if n == 0 else F.gelu(x))
        loss = F.cross_entropy(x, y)
        params = [p for layer in layers for p in layer.parameters()]
        grads = list(torch.autograd.grad(loss, params))
        weights = [p.detach() for p in params]
        _adamw64(weights, grads, [(torch.zeros_like(p), torch.zeros_like(p)) for p in weights], 1)
        return {"loss": loss.detach(), "weights": weights, "grads": grads}
    ws, n = case["ranks"], case["n"]
    count = n * ws if case["op"] == "reduce_scatter" else n
    ins = [torch.randn(count, generator=gen, device=device).to(_DTYPES[case["dtype"]]).double() for _ in range(ws)]
    if case["op"] == "allreduce":
        return [sum(ins) / ws] * ws
    if case["op"] == "reduce_scatter":
        return list((sum(ins) / ws).chunk(ws))
    if case["op"] == "allgather":
        return [torch.cat(ins)] * ws
    return [ins[0]] * ws
