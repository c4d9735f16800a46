"""The fp32 linear layer on the tensor cores against the same products in 64 bits."""
import copy
import gc
import subprocess
import sys
import threading
import time
from pathlib import Path

import pytest
import torch
import torch.distributed as dist
import torch.nn.functional as F

import mccl_b200
from mccl_b200.models import MLP94M
from mccl_b200.ops.linear import Linear, linear
from mccl_b200.parallel import wrap_ddp


def _bound(absolute, depth):
    """What may separate a product from its value: three parts leave 2^-24 of every factor out, the tensor cores cut off
    (2^-23 of the running sum) each of the at most 8 sums of 16 products between two rounded additions, and the additions
    of the depth / 64 parts round by 2^-24 each.  `absolute`: the product of the absolute values."""
    return absolute * (2.0 ** -20 + (depth / 64 + 2) * 2.0 ** -24)


# rows around the tiles of 32, 64 and 128; features that are no multiple of anything; split and unsplit reductions
@pytest.mark.gpu
@pytest.mark.parametrize("batch,n_in,n_out", [
    (8, 3072, 3072), (32, 1027, 1001), (33, 1001, 1027), (64, 1500, 1500), (65, 1237, 1300), (100, 1100, 1000),
    (127, 3071, 1000), (128, 1024, 1024), (129, 1023, 1025), (255, 2048, 3000), (256, 3072, 3072), (700, 1000, 2100),
])
def test_linear_matches_64_bits(batch, n_in, n_out):
    native = mccl_b200.require_native()
    torch.manual_seed(batch)
    x = torch.randn(batch, n_in, device="cuda", requires_grad=True)
    w = torch.randn(n_out, n_in, device="cuda", requires_grad=True)
    b = torch.randn(n_out, device="cuda", requires_grad=True)
    g = torch.randn(batch, n_out, device="cuda")
    assert native._linear_native(x, w, b)
    y = linear(x, w, b)
    got = [y, *torch.autograd.grad(y, (x, w, b), g)]
    x, w, b, g = (t.detach().double() for t in (x, w, b, g))
    want = [x @ w.T + b, g @ w, g.T @ x, g.sum(0)]
    size = [x.abs() @ w.abs().T + b.abs(), g.abs() @ w.abs(), g.abs().T @ x.abs(), g.abs().sum(0)]
    for name, a, r, s, depth in zip("y x w b".split(), got, want, size, (n_in, n_out, batch, batch)):
        assert ((a.detach().double() - r).abs() <= _bound(s, depth)).all(), name


# views: rows of a wider matrix, a start that is off 16 bytes, a gradient that is a transposed or expanded view
@pytest.mark.gpu
@pytest.mark.parametrize("shift,pad", [(0, 0), (0, 4), (1, 3), (3, 1), (0, 5)])
def test_linear_of_views(shift, pad):
    torch.manual_seed(0)
    batch, n_in, n_out = 130, 1004, 1100

    def view(rows, cols):
        return torch.randn(rows, cols + shift + pad, device="cuda")[:, shift:shift + cols]

    x, w = view(batch, n_in).requires_grad_(), view(n_out, n_in).requires_grad_()
    assert mccl_b200.require_native()._linear_native(x, w, None)
    for g in (view(batch, n_out), view(n_out, batch).T, torch.randn(1, n_out, device="cuda").expand(batch, n_out)):
        y = linear(x, w)
        got = [y, *torch.autograd.grad(y, (x, w), g)]
        xd, wd, gd = (t.detach().double() for t in (x, w, g))
        for a, r, s, depth in ((got[0], xd @ wd.T, xd.abs() @ wd.abs().T, n_in),
                               (got[1], gd @ wd, gd.abs() @ wd.abs(), n_out),
                               (got[2], gd.T @ xd, gd.abs().T @ xd.abs(), batch)):
            assert ((a.detach().double() - r).abs() <= _bound(s, depth)).all()


@pytest.mark.gpu
def test_linear_special_values():
    """Infinities, NaN and the largest and smallest normal numbers go through as in a multiplication."""
    torch.manual_seed(0)
    x, w = torch.randn(64, 1024, device="cuda"), torch.randn(1024, 1024, device="cuda")
    x[0, 5], x[1, 6], x[2, 7], w[3, 9], w[4, 10] = float("inf"), float("nan"), -float("inf"), float("inf"), float("nan")
    x[5, 20], w[6, 21] = 3.4028234e38, -3.4028234e38
    w[:, 5] = torch.where(w[:, 5].abs() < 0.1, 0.0, w[:, 5])  # inf * 0
    x[7], w[:, 20] = x[7] * 1e-37, w[:, 20] * 1e-3
    x[8, 6] = torch.tensor(0x7F800001, dtype=torch.int32).view(torch.float32).item()  # a NaN in its last bit alone
    got, want = linear(x, w), F.linear(x, w)
    assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
    assert torch.equal(got[got.isinf()], want[want.isinf()])
    exact = x.double() @ w.double().T
    ok = want.isfinite()
    bound = _bound(x.double().abs() @ w.double().abs().T, 1024)
    assert ((got.double() - exact).abs()[ok] <= bound[ok]).all()


# Error of whole products, 2-norm against 64 bits.  A result is the sum of a group of 64 of the reduction after the other, each rounded
# to fp32, and the tensor cores cut their sums off at each of a group's four steps: at most some 4 units of 2^-24 of the partial
# sums, which are no larger than the result's own size.  Without the least of the six products (2^-17 of a number) it is 7e-6.
# Each tile width, split and unsplit reductions, several tiles per CTA forward and for the input gradient, ragged edges.
@pytest.mark.gpu
@pytest.mark.parametrize("batch,n_in,n_out", [(24, 1500, 1340), (32, 3072, 3072), (50, 1700, 1027), (64, 2048, 2048),
                                              (100, 1030, 1410), (256, 3072, 3072), (700, 1000, 4100), (2000, 3000, 2900)])
def test_linear_error_of_whole_products(batch, n_in, n_out):
    torch.manual_seed(batch)
    x = torch.randn(batch, n_in, device="cuda", requires_grad=True)
    w = (torch.randn(n_out, n_in, device="cuda") / n_in ** 0.5).requires_grad_()
    b, g = torch.randn(n_out, device="cuda", requires_grad=True), torch.randn(batch, n_out, device="cuda")
    assert mccl_b200.require_native()._linear_native(x, w, b)
    y = linear(x, w, b)
    grads = torch.autograd.grad(y, (x, w, b), g)
    x, w, b, g = (t.detach().double() for t in (x, w, b, g))
    for got, want in zip((y, *grads), (x @ w.T + b, g @ w, g.T @ x, g.sum(0))):
        assert (got.double() - want).norm() <= 4 * 2.0 ** -24 * want.norm()


def _floats(gen, rows, cols, exponent):
    """Positive floats of one power of two whose lower 16 bits, what the leading bf16 part leaves, are of every size."""
    upper = torch.randint(0, 128, (rows, cols), generator=gen) << 16
    lower = torch.where(torch.rand(rows, cols, generator=gen) < 0.5, torch.randint(0, 65536, (rows, cols), generator=gen),
                        torch.randint(0x7F00, 0x8100, (rows, cols), generator=gen) ^ 0x8000)
    return (((exponent + 127) << 23) | upper | lower).int().view(torch.float32)


# One non-zero per row of the input: every result is one product, in the left-over terms and the range of which nothing hides.
# Left out: mid lo + lo mid + lo lo with |mid| <= 2^-8 and |lo| <= 2^-17 of the power of two of its number: 2^-24 (1 + 2^-10) of
# the product.  Joining the accumulators rounds twice, 2^-24 of the result and 2^-24 of its part below 2^-7; 2^-29 for sums cut off.
@pytest.mark.gpu
@pytest.mark.parametrize("batch,exponents", [(32, (0, 0)), (64, (3, -60)), (128, (0, 127)), (64, (63, 63)), (32, (127, 0)),
                                             (64, (64, 63))])
def test_linear_of_single_products(batch, exponents):
    gen = torch.Generator().manual_seed(batch)
    x = torch.zeros(batch, 1024)
    at = torch.arange(batch)
    x[at, 7 * at] = _floats(gen, batch, 1, exponents[0])[:, 0] * torch.where(at % 2 == 0, 1.0, -1.0)
    w = _floats(gen, 1024, 1024, exponents[1])
    w[0] = (2 - 2.0 ** -23) * 2.0 ** exponents[1]  # for an exponent of 127 the largest number there is
    assert mccl_b200.require_native()._linear_native(x.cuda(), w.cuda(), None)
    got = linear(x.cuda(), w.cuda()).cpu().double()
    want = x[at, 7 * at].double()[:, None] * w.T[7 * at].double()
    most = torch.finfo(torch.float32).max
    fits = want.abs() <= most * (1 - 2.0 ** -23)
    bound = want.abs() * 2.0 ** -24 * (2 + 2.0 ** -5)
    assert ((got - want).abs() <= bound)[fits].all(), ((got - want).abs() / bound)[fits].max()
    over = want.abs() >= most * (1 + 2.0 ** -23)
    assert got[over].isinf().all() and torch.equal(got[over].sign(), want[over].sign())
    if sum(exponents) < 126:
        assert fits.all()
    elif sum(exponents) < 127:
        assert fits.any()


@pytest.mark.gpu
def test_linear_keeps_what_autograd_offers():
    torch.manual_seed(0)
    x = torch.randn(64, 1024, device="cuda", requires_grad=True)
    layer = Linear(1024, 1024).cuda()
    w, b = layer.weight, layer.bias

    def both(fn):
        torch.testing.assert_close(fn(linear), fn(F.linear), rtol=1e-4, atol=1e-3)

    def second(f):
        (g,) = torch.autograd.grad(f(x, w, b).square().sum(), x, create_graph=True)
        return torch.autograd.grad(g.square().sum(), w)[0] * 1e-4

    both(second)
    both(lambda f: torch.func.jvp(lambda t: f(t, w, b), (x,), (x,))[1])
    both(lambda f: torch.func.vmap(lambda t: f(t, w, b))(x.expand(2, 64, 1024)))
    both(lambda f: torch.func.grad(lambda t: f(x, t, b).square().sum())(w) * 1e-3)
    both(lambda f: torch.autograd.grad(f(x, w, b), x, torch.ones(3, 64, 1024, device="cuda"), is_grads_batched=True)[0])
    both(lambda f: torch.autograd.grad(f(x, w, b).sum(), b)[0])
    packed = []
    with torch.autograd.graph.saved_tensors_hooks(lambda t: packed.append(t.shape) or t, lambda t: t):
        linear(x, w, b).sum().backward()
    assert packed == [x.shape, w.shape] and layer.weight.grad is not None
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert layer(x).dtype == torch.bfloat16
    y = layer(x).sum()
    with torch.no_grad():
        w.add_(1.0)
    with pytest.raises(RuntimeError, match="modified by an inplace operation"):
        y.backward()
    stock = copy.deepcopy(layer)
    stock.stock = True
    assert torch.equal(stock(x), F.linear(x, w, b))


@pytest.mark.gpu
def test_linear_under_capture_and_streams():
    x, w = torch.randn(64, 2048, device="cuda"), torch.randn(1000, 2048, device="cuda")
    want = linear(x, w)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        other = linear(x, w)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = linear(x, w)
    for _ in range(2):
        y.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want) and torch.equal(other, want)


# A wait that runs out: the kernel ends by itself, everything it should have written is NaN, the next call on the device says so
# once, and then the layer works as before.  Split and unsplit reductions, one and several tiles per CTA, each tile width.
@pytest.mark.gpu
@pytest.mark.parametrize("batch,n_in,n_out", [(32, 3072, 3072), (64, 1500, 1500), (256, 3072, 3072), (700, 1000, 4100),
                                              (2000, 3000, 2900)])
def test_linear_whose_waits_run_out(batch, n_in, n_out):
    native = mccl_b200.require_native()
    torch.manual_seed(0)
    x, w, g = (torch.randn(*s, device="cuda") for s in ((batch, n_in), (n_out, n_in), (batch, n_out)))
    want = linear(x, w)
    (out,) = native._linear_with_limit(x, w, None, 0)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="a wait inside"):
        linear(x, w)
    assert out.isnan().all()
    assert torch.equal(linear(x, w), want)
    outs = native._linear_with_limit(x, w, g, 0)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError, match="a wait inside"):
        linear(x, w)
    own = [t.isnan().any().item() for t in outs]  # a product that does not pay is the library's
    assert any(own) and all(t.isnan().all() for t, o in zip(outs, own) if o)
    assert torch.equal(linear(x, w), want)


@pytest.mark.gpu
@pytest.mark.parametrize("setting", ["torch.backends.cuda.matmul.fp32_precision = 'tf32'", "torch.backends.fp32_precision = 'tf32'",
                                     "torch.set_float32_matmul_precision('high')", "torch.backends.cuda.matmul.allow_tf32 = True"])
def test_linear_where_tf32_is_allowed(setting):
    """Each way to allow it leaves the products to torch (in a process of its own: the settings do not mix)."""
    code = f"""
import torch, torch.nn.functional as F, mccl_b200
from mccl_b200.ops.linear import linear
x, w = torch.randn(64, 2048, device="cuda"), torch.randn(2048, 2048, device="cuda")
native = mccl_b200.require_native()
assert native._linear_native(x, w, None)
{setting}
assert not native._linear_native(x, w, None)
assert torch.equal(linear(x, w), F.linear(x, w))
"""
    done = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parents[1], capture_output=True, text=True)
    assert done.returncode == 0, done.stderr[-2000:]


@pytest.mark.gpu
def test_linear_without_memory_for_its_images():
    """Where the images cannot be had the products are torch's."""
    native = mccl_b200.require_native()
    torch.manual_seed(0)
    batch, n_in, n_out = 8192, 4096, 2048  # images of 201 MB forward and of 302 MB backward, tensors of 134, 67 and 34 MB
    x, w, g = (torch.randn(*s, device="cuda", requires_grad=s[1] == n_in) for s in ((batch, n_in), (n_out, n_in), (batch, n_out)))
    assert native._linear_native(x, w, None)
    torch.cuda.empty_cache()
    _, total = torch.cuda.mem_get_info()
    try:
        y = linear(x, w)
        torch.cuda.empty_cache()
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (190 << 20)) / total)
        with torch.no_grad():
            z = linear(x, w)
        assert torch.equal(z, F.linear(x, w)) and not torch.equal(z, y)
        del z
        torch.cuda.empty_cache()
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (280 << 20)) / total)
        gx, gw = torch.autograd.grad(y, (x, w), g)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
        torch.cuda.empty_cache()
    assert torch.equal(gx, g.mm(w)) and torch.equal(gw, g.t().mm(x))


class _Seen(torch.Tensor):
    """A subclass that sees the functions it is passed to."""

    @classmethod
    def __torch_function__(cls, func, types, args=(), kwargs=None):
        cls.seen = func
        return super().__torch_function__(func, types, args, kwargs or {})


@pytest.mark.gpu
@pytest.mark.parametrize("which", [0, 1, 2])
def test_linear_of_subclasses(which):
    args = [torch.randn(64, 1024, device="cuda"), torch.randn(1024, 1024, device="cuda"), torch.randn(1024, device="cuda")]
    args[which] = args[which].as_subclass(_Seen)
    _Seen.seen = None
    assert type(linear(*args)) is _Seen and _Seen.seen is F.linear


# Measured (B200): what the library does faster by a quarter and more stays its own, what it does slower by a tenth and more does not.
# Rows, features in and out.
@pytest.mark.parametrize("product,ours,library", [
    ("forward", [(8, 3072, 3072), (64, 512, 2048), (256, 3072, 3072), (200, 512, 3000), (96, 1024, 700), (32, 16384, 128),
                 (4, 8192, 1000), (64, 1024, 50257), (4096, 4096, 4096)],
     [(64, 65536, 16), (64, 100000, 64), (16, 16384, 128), (16, 32768, 256), (1, 8192, 8192), (2, 4096, 16384), (4, 1024, 50257),
      (96, 256, 3000), (128, 400, 2048), (128, 300, 4000), (128, 16, 65536), (1, 700000, 1)]),
    ("input", [(8, 3072, 3072), (256, 3072, 3072), (64, 1024, 1024), (256, 2048, 1000), (2, 8192, 8192), (128, 1400, 1400),
               (512, 16384, 128)],
     [(64, 65536, 16), (256, 16, 65536), (16, 128, 16384), (128, 64, 65536), (1, 8192, 8192), (1, 1024, 50257), (4, 32768, 256),
      (96, 3000, 256)]),
    ("weight", [(256, 3072, 3072), (64, 2048, 1000), (96, 850, 1400), (200, 400, 3000), (128, 1024, 1400)],
     [(256, 65536, 16), (512, 100000, 64), (256, 64, 65536), (16, 3072, 3072)]),
])
def test_linear_takes_what_it_does_faster(product, ours, library):
    pays = mccl_b200.require_native()._linear_pays
    assert all(pays(product, *s) for s in ours) and not any(pays(product, *s) for s in library)


def test_linear_lets_other_threads_run():
    native = mccl_b200.require_native()
    x, w = torch.randn(4096, 4096), torch.randn(4096, 4096)
    done, ticks = threading.Event(), set()

    def call():
        for _ in range(4):
            native._linear(x, w, None)
        done.set()

    begin = time.monotonic()
    thread = threading.Thread(target=call)
    thread.start()
    while not done.wait(0.001):
        ticks.add(int((time.monotonic() - begin) * 100))
    took = time.monotonic() - begin
    thread.join()
    assert len(ticks) > 0.3 * 100 * took  # hundredths of a second in which this thread ran, too


def test_linear_elsewhere_is_torch():
    """What the kernels do not take is torch's own call: other devices, types and orders, scripting and tracing."""
    native = mccl_b200.require_native()
    torch.manual_seed(0)
    for dtype in (torch.float32, torch.float64, torch.bfloat16):
        x, w, b = (torch.randn(*s).to(dtype) for s in ((4, 64, 48), (32, 48), (32,)))
        for xi in (x, x[0], x[0, 0], x[0, :, ::2].expand(64, 24)):
            wi = w[:, :xi.shape[-1]]
            assert not native._linear_native(xi, wi, b)
            assert torch.equal(native._linear(xi, wi, b), F.linear(xi, wi, b))
            assert torch.equal(linear(xi, wi), F.linear(xi, wi))
    model = MLP94M(64, 48, 1, 5)
    x = torch.randn(3, 64)
    assert torch.equal(torch.jit.script(model)(x), model(x)) and torch.equal(torch.jit.trace(model, x)(x), model(x))
    assert torch.equal(torch.fx.symbolic_trace(model)(x), model(x))
    assert all(isinstance(m, torch.nn.Linear) for m in model.net[::2])
    assert list(model.state_dict())[:2] == ["net.0.weight", "net.0.bias"]
    with pytest.raises(RuntimeError):
        linear(torch.randn(3, 5), torch.randn(4, 6))


@pytest.mark.gpu
def test_compressed_wrapper_gives_its_layers_back():
    """A module keeps torch's products while a compressed wrapper of it lives, and no longer; the program's own choice stays."""
    created = not dist.is_initialized()
    if created:
        dist.init_process_group("mccl", store=dist.HashStore(), rank=0, world_size=1)
    try:
        model = MLP94M(64, 48, 1, 5).cuda()
        layers = model.net[::2]
        layers[0].stock = True
        own = lambda: [not m.stock for m in layers]  # noqa: E731
        first = wrap_ddp(model, device_ids=[0], compression="topk")
        assert own() == [False, False, False]
        dense = wrap_ddp(model, device_ids=[0], compression="none")
        assert own() == [False, True, True]
        second = wrap_ddp(model, device_ids=[0], compression="topk")
        assert own() == [False, False, False]
        del first, dense
        gc.collect()
        assert own() == [False, False, False]
        del second
        gc.collect()
        assert own() == [False, True, True]
        assert torch.equal(layers[0](torch.ones(2, 64, device="cuda")),
                           F.linear(torch.ones(2, 64, device="cuda"), layers[0].weight, layers[0].bias))
    finally:
        if created:
            dist.destroy_process_group()
