"""STFT / iSTFT kernels vs torch.stft / torch.istft on the CPU (the oracle).

Mirrors the reference's tests/test_stft_vdsp.py:22-124: forward parity < 1e-4, gradient
agreement, finite inverse, and a wall-clock guard for forward+backward.
"""
import time

import pytest
import torch

import mccl_b200
from mccl_b200.transforms import istft, resolve_backend, stft


def test_backend_names():
    assert resolve_backend("metal") == "cuda" and resolve_backend("vdsp") == "cpu" and resolve_backend("auto") == "auto"
    with pytest.raises(ValueError):
        resolve_backend("fftw")


def test_cpu_backend_matches_torch():
    x = torch.randn(2, 4000)
    w = torch.hann_window(512)
    got = stft(x, n_fft=512, hop_length=128, win_length=512, window=w, backend="vdsp")
    ref = torch.stft(x, 512, hop_length=128, win_length=512, window=w, center=True, return_complex=True)
    assert torch.allclose(got, ref)


def _cos(a, b):
    a, b = a.flatten().double(), b.flatten().double()
    return float((a @ b) / (a.norm() * b.norm() + 1e-30))


@pytest.mark.gpu
@pytest.mark.parametrize("n_fft,hop,win", [(2048, 512, 2048), (1024, 256, 1024), (512, 128, 400), (64, 16, 64)])
@pytest.mark.parametrize("center", [True, False])
@pytest.mark.parametrize("normalized", [False, True])
def test_stft_forward_and_backward_match_torch(cuda_device, n_fft, hop, win, center, normalized):
    torch.manual_seed(0)
    x = torch.randn(2, 48000 if n_fft > 64 else 1000)
    w = torch.hann_window(win, periodic=True)
    kw = dict(n_fft=n_fft, hop_length=hop, win_length=win)
    xr = x.clone().requires_grad_(True)
    ref = torch.stft(xr, window=w, center=center, normalized=normalized, return_complex=True, **kw)
    xg = x.to(cuda_device).requires_grad_(True)
    got = stft(xg, window=w.to(cuda_device), center=center, normalized=normalized, backend="cuda", **kw)
    assert got.shape == ref.shape
    assert float((ref - got.detach().cpu()).abs().max()) < 1e-4 * max(1.0, float(ref.abs().max()) / 30)
    # gradient of a generic real loss
    gr = torch.randn(ref.shape, dtype=torch.complex64)
    (ref * gr.conj()).real.sum().backward()
    (got * gr.to(cuda_device).conj()).real.sum().backward()
    assert _cos(xg.grad.cpu(), xr.grad) > 0.9999
    assert torch.allclose(xg.grad.cpu(), xr.grad, rtol=1e-3, atol=1e-3 * float(xr.grad.abs().max()))


@pytest.mark.gpu
@pytest.mark.parametrize("n_fft,hop", [(1024, 256), (512, 128), (2048, 512)])
@pytest.mark.parametrize("normalized", [False, True])
def test_istft_forward_and_backward_match_torch(cuda_device, n_fft, hop, normalized):
    torch.manual_seed(1)
    length = 24000
    w = torch.hann_window(n_fft, periodic=True)
    x = torch.randn(2, length)
    spec = torch.stft(x, n_fft, hop_length=hop, win_length=n_fft, window=w, center=True, normalized=normalized,
                      return_complex=True)
    spec = spec + 0.1 * torch.randn_like(spec)  # not exactly consistent: exercises the general case
    sr = spec.clone().requires_grad_(True)
    ref = torch.istft(sr, n_fft, hop_length=hop, win_length=n_fft, window=w, center=True, normalized=normalized,
                      length=length)
    sg = spec.to(cuda_device).requires_grad_(True)
    got = istft(sg, n_fft=n_fft, hop_length=hop, win_length=n_fft, window=w.to(cuda_device), length=length,
                normalized=normalized, backend="cuda")
    assert torch.isfinite(got).all()
    assert float((ref - got.detach().cpu()).abs().max()) < 1e-4
    gy = torch.randn(ref.shape)
    (ref * gy).sum().backward()
    (got * gy.to(cuda_device)).sum().backward()
    # compare only what an inverse real FFT can see (imaginary DC/Nyquist parts have no gradient)
    assert _cos(sg.grad.cpu().real, sr.grad.real) > 0.9999
    a, b = torch.view_as_real(sg.grad.cpu()), torch.view_as_real(sr.grad)
    assert torch.allclose(a, b, rtol=1e-3, atol=1e-3 * float(b.abs().max()))


@pytest.mark.gpu
def test_roundtrip_and_perf_guard(cuda_device):
    w = torch.hann_window(2048, device=cuda_device)
    x = torch.randn(2, 48000, device=cuda_device, requires_grad=True)
    kw = dict(n_fft=2048, hop_length=512, win_length=2048, window=w)
    for _ in range(2):  # warm-up
        stft(x, **kw).abs().sum().backward()
    torch.cuda.synchronize()
    t0 = time.perf_counter()
    s = stft(x, **kw)
    y = istft(s, length=48000, **kw)
    (y.square().sum() + s.abs().sum()).backward()
    torch.cuda.synchronize()
    assert (time.perf_counter() - t0) * 1e3 < 1000  # the reference's guard: fwd+bwd under one second
    assert float((y.detach() - x.detach()).abs().max()) < 1e-3  # hann/4-overlap satisfies the NOLA condition


@pytest.mark.gpu
def test_rejects_unsupported_sizes(cuda_device):
    x = torch.randn(1, 5000, device=cuda_device)
    with pytest.raises(ValueError):
        stft(x, n_fft=1000, hop_length=250, win_length=1000, window=torch.hann_window(1000, device=cuda_device),
             backend="cuda")
    # "auto" falls back to ATen for sizes the kernels do not cover
    out = stft(x, n_fft=1000, hop_length=250, win_length=1000, window=torch.hann_window(1000, device=cuda_device))
    assert out.shape[1] == 501


def _rel(got, ref):
    got, ref = got.detach().cpu(), ref.detach()
    return float((got - ref).norm() / ref.norm())


# Every transform length, frames that fill a warp or leave lanes without one, one segment or many, odd lengths (rows off
# an 8-byte boundary), hops that do not divide n_fft, hops so small that the inverse takes its two-kernel path, and
# signals at and below the length from which the folded edges are disjoint (n_fft + 2).
@pytest.mark.gpu
@pytest.mark.parametrize("n_fft,hop,samples,batch", [
    (8, 2, 61, 3), (8, 4, 10, 1), (16, 4, 1001, 2), (16, 1, 77, 2), (32, 8, 4099, 1), (64, 20, 999, 3),
    (128, 32, 30011, 2), (256, 80, 20001, 5), (512, 128, 16000, 1), (512, 512, 5000, 2), (1024, 256, 1025, 2),
    (1024, 256, 1026, 2), (1024, 320, 120007, 3), (1024, 16, 9001, 1), (2048, 512, 1030, 2), (2048, 512, 300001, 4),
    (4096, 1024, 4098, 1), (4096, 1024, 200003, 2), (4096, 1280, 50001, 2)])
@pytest.mark.parametrize("frames_major", [True, False])
def test_transforms_match_float64(cuda_device, n_fft, hop, samples, batch, frames_major):
    gen = torch.Generator().manual_seed(n_fft + hop)
    win_len = n_fft - n_fft // 8
    w = 0.1 + torch.rand(win_len, generator=gen)  # asymmetric, no zeros inside
    x = torch.randn(batch, samples, generator=gen)
    kw = dict(n_fft=n_fft, hop_length=hop, win_length=win_len)
    frames = 1 + samples // hop
    g = torch.randn(batch, n_fft // 2 + 1, frames, dtype=torch.complex64, generator=gen)
    spec = torch.randn(batch, n_fft // 2 + 1, frames, dtype=torch.complex64, generator=gen)
    # relative to the norm of the whole result: log2(n_fft) + 1 <= 13 roundings of 6e-8 in the transform, a few more
    # for the table entries, the window and the sum of the overlapping frames; they add up as a random walk
    tol = 6e-8 * 16

    def layout(t):  # same values; memory order frames-major (the framework's own) or bins-major (a network's output)
        return t.transpose(1, 2).contiguous().transpose(1, 2) if frames_major else t.contiguous()

    xd = x.double().requires_grad_(True)
    ref = torch.stft(xd, window=w.double(), center=True, return_complex=True, **kw)
    (ref_g,) = torch.autograd.grad(ref, xd, g.to(torch.complex128))
    xc = x.to(cuda_device).requires_grad_(True)
    out = stft(xc, window=w.to(cuda_device), backend="cuda", **kw)
    (out_g,) = torch.autograd.grad(out, xc, layout(g.to(cuda_device)))
    assert _rel(out, ref) < tol
    assert _rel(out_g, ref_g) < tol

    # the inverse over samples that some frame covers (win_len < n_fft leaves gaps when hop > win_len); its gradient
    length = min(samples, (frames - 1) * hop)
    if hop <= win_len and length > 0:
        sd = spec.to(torch.complex128).requires_grad_(True)
        inv = torch.istft(sd, window=w.double(), center=True, length=length, **kw)
        (inv_g,) = torch.autograd.grad(inv, sd, x.double()[:, :length])
        sc = layout(spec.to(cuda_device)).requires_grad_(True)
        got = istft(sc, window=w.to(cuda_device), length=length, backend="cuda", **kw)
        (got_g,) = torch.autograd.grad(got, sc, x.to(cuda_device)[:, :length])
        assert _rel(got, inv) < tol
        assert _rel(got_g, inv_g) < tol


@pytest.mark.gpu
@pytest.mark.parametrize("length", [3000, 20000])  # shorter and far longer than what the frames cover
def test_istft_beyond_the_frames_is_zero(cuda_device, length):
    spec = torch.randn(2, 129, 100, dtype=torch.complex64, device=cuda_device)
    w = torch.ones(256, device=cuda_device)
    full = istft(spec, n_fft=256, hop_length=64, win_length=256, window=w, length=64 * 99 + 128, backend="cuda")
    got = istft(spec, n_fft=256, hop_length=64, win_length=256, window=w, length=length, backend="cuda")
    keep = min(length, full.shape[1])
    assert torch.equal(got[:, :keep], full[:, :keep])
    assert not got[:, keep:].any()


# Lazy views: `.conj()` only sets a bit, and autograd hands such tensors to backward as well; `.conj().imag` sets the
# negative bit.  The transforms have to see the values, in both memory orders.
@pytest.mark.gpu
@pytest.mark.parametrize("frames_major", [True, False])
def test_lazily_conjugated_and_negated_inputs(cuda_device, frames_major):
    n_fft, hop, samples = 256, 64, 4001
    gen = torch.Generator().manual_seed(9)
    w = torch.hann_window(n_fft)
    kw = dict(n_fft=n_fft, hop_length=hop, win_length=n_fft)
    z = torch.randn(2, samples, dtype=torch.complex64, generator=gen)
    spec = torch.randn(2, n_fft // 2 + 1, 1 + samples // hop, dtype=torch.complex64, generator=gen)
    dev_spec = spec.to(cuda_device)
    if frames_major:
        dev_spec = dev_spec.transpose(1, 2).contiguous().transpose(1, 2)
    tol = 6e-8 * 16

    def reference(fn):  # fn on float64 host tensors, with torch's own transforms
        return fn(lambda t: torch.stft(t, window=w.double(), return_complex=True, **kw),
                  lambda s, n: torch.istft(s, window=w.double(), length=n, **kw), z.to(torch.complex128), spec.to(torch.complex128))

    def ours(fn):
        wd = w.to(cuda_device)
        return fn(lambda t: stft(t, window=wd, backend="cuda", **kw),
                  lambda s, n: istft(s, window=wd, length=n, backend="cuda", **kw), z.to(cuda_device), dev_spec)

    length = (spec.shape[2] - 1) * hop

    def inverse(fwd, inv, z, s):
        return inv(s.conj(), length)

    def negated_waveform(fwd, inv, z, s):
        return fwd(z.conj().imag)

    def gradient_through_conj(fwd, inv, z, s):
        x = z.real.clone().requires_grad_(True)
        return torch.autograd.grad(fwd(x).conj(), x, s)[0]

    def gradient_of_inverse_through_conj(fwd, inv, z, s):
        s = s.detach().clone().requires_grad_(True)
        return torch.autograd.grad(inv(s.conj(), length), s, z.conj().imag[:, :length])[0]

    for fn in (inverse, negated_waveform, gradient_through_conj, gradient_of_inverse_through_conj):
        assert _rel(ours(fn), reference(fn)) < tol, fn.__name__


# A spectrum (or its gradient) with any strides: expanded over the batch, sliced in every dimension, one frame or bin
# repeated by a zero stride.  The same values give the same bits whatever the strides.
@pytest.mark.gpu
def test_transforms_follow_the_spectrum_strides(cuda_device):
    n_fft, hop, samples = 512, 128, 9001
    frames, bins = 1 + samples // hop, n_fft // 2 + 1
    gen = torch.Generator(device=cuda_device).manual_seed(3)
    w = torch.hann_window(n_fft, device=cuda_device)
    kw = dict(n_fft=n_fft, hop_length=hop, win_length=n_fft, window=w, backend="cuda")

    def rand(*shape):
        return torch.randn(*shape, dtype=torch.complex64, generator=gen, device=cuda_device)

    views = [rand(1, bins, frames).expand(3, -1, -1), rand(3, 1, frames).expand(-1, bins, -1),
             rand(3, bins, 1).expand(-1, -1, frames), rand(6, 2 * bins, 3 * frames)[::2, 1::2, 2::3],
             rand(frames, bins, 3).permute(2, 1, 0), rand(3, frames, bins + 5)[:, :, 3:-2].transpose(1, 2),
             rand(1, 1, 1).expand(3, bins, frames)]
    x = torch.randn(3, samples, generator=gen, device=cuda_device, requires_grad=True)
    for v in views:
        assert v.shape == (3, bins, frames)
        for plain in (v.contiguous(), v.transpose(1, 2).contiguous().transpose(1, 2)):
            assert torch.equal(istft(v, length=samples, **kw), istft(plain, length=samples, **kw))
            got, want = (torch.autograd.grad(stft(x, **kw), x, g)[0] for g in (v, plain))
            assert torch.equal(got, want)


# A hop far beyond the signal, up to and beyond the range of an int: one frame, whatever the hop.
@pytest.mark.gpu
@pytest.mark.parametrize("hop", [1_000_000, 2**30 + 1, 2**31 - 4000, 2**31 - 1, 2**31, 2**32, 2**33 + 7])
@pytest.mark.parametrize("n_fft", [8, 1024, 4096])
def test_hops_beyond_the_signal(cuda_device, n_fft, hop):
    samples, length = 3 * n_fft, n_fft // 2
    gen = torch.Generator(device=cuda_device).manual_seed(5)
    w = 0.1 + torch.rand(n_fft, generator=gen, device=cuda_device)
    x = torch.randn(2, samples, generator=gen, device=cuda_device, requires_grad=True)
    spec = torch.randn(2, n_fft // 2 + 1, 1, dtype=torch.complex64, generator=gen, device=cuda_device, requires_grad=True)

    def all_four(h):
        kw = dict(n_fft=n_fft, hop_length=h, win_length=n_fft, window=w, backend="cuda")
        out, back = stft(x, **kw), istft(spec, length=length, **kw)
        return (out, torch.autograd.grad(out, x, spec.detach())[0], back,
                torch.autograd.grad(back, spec, x.detach()[:, :length])[0])

    for got, want in zip(all_four(hop), all_four(samples + 1)):
        assert torch.equal(got, want)


# The fused inverse cuts the output into segments of rows, one per CTA.  Every row once and in order; a folded edge within one
# segment; and no segment with more batches of frames than the longest of an even cut would need (a row or two too many
# cost calls of few frames a second batch).
@pytest.mark.parametrize("n_fft,hop", [(8, 2), (64, 20), (256, 64), (512, 128), (1024, 256), (1024, 320), (2048, 512), (2048, 1024),
                                       (2048, 2048), (1024, 128), (4096, 1024), (4096, 1280), (4096, 3000)])
@pytest.mark.parametrize("fold", [True, False])
def test_inverse_segments(native, n_fft, hop, fold):
    for batch in (1, 2, 5, 16, 400):
        for frames in list(range(1, 40)) + [64, 94, 95, 188, 313, 1000, 2049, 20001]:
            length = max(1, (frames - 1) * hop + (hop * 3) // 7)
            reach, together, most, begins = native._test_stft_inverse_shape(n_fft, hop, length, frames, batch, fold)
            if not begins:
                assert fold and length < n_fft + 2
                continue
            first = 0 if fold else (n_fft // 2) // hop
            end = -(-(length + (n_fft if fold else n_fft // 2)) // hop)
            assert begins[0] == first and begins[-1] == end
            sizes = [b - a for a, b in zip(begins, begins[1:])]
            assert min(sizes) >= 1
            if fold and len(sizes) > 1:
                assert min(sizes[0], sizes[-1]) >= reach + 1
            assert len(sizes) <= most + 2

            def batches(lo, hi):
                return -(-max(0, min(hi, frames) - max(0, lo - reach + 1)) // together)

            even = -(-(end - first) // most)          # rows
            bound = -(-(even + reach - 1) // together)
            # a segment that has to hold a folded edge may need one more
            edges = -(-(reach + 1) // together) if fold else 0
            assert max(batches(a, b) for a, b in zip(begins, begins[1:])) <= max(bound, edges) or len(sizes) == 1


# the one native call against the Python functions that it stands in for: bit for bit, over the forms that both take
@pytest.mark.gpu
@pytest.mark.parametrize("shape,dtype,window_grad", [((4000,), torch.float32, False), ((2, 4001), torch.float32, False),
                                                     ((2, 1, 4001), torch.float32, True), ((3, 4000), torch.bfloat16, False)])
def test_direct_calls_match_the_functions(shape, dtype, window_grad):
    from mccl_b200.transforms import stft as module_fn  # noqa: F401  (the package exports the functions)
    import importlib
    mod = importlib.import_module("mccl_b200.transforms.stft")
    torch.manual_seed(0)
    x = torch.randn(*shape, device="cuda").to(dtype).requires_grad_()
    win = torch.hann_window(400, device="cuda").requires_grad_(window_grad)
    kw = dict(n_fft=512, hop_length=128, win_length=400, window=win)
    native = mod.require_native()
    got = mod.stft(x, **kw)
    want = mod._StftFn.apply(x, win, 512, 128, 400, True, False)
    g = torch.randn_like(want)
    assert torch.equal(got, want) and got.requires_grad and got.stride() == want.stride()
    assert torch.equal(torch.autograd.grad(got, x, g)[0], torch.autograd.grad(want, x, g)[0])
    spec = want.detach().requires_grad_()
    got = mod.istft(spec, length=4000, **kw)
    want = mod._IstftFn.apply(spec, win, 512, 128, 400, 4000, True, False)
    g = torch.randn_like(want)
    assert torch.equal(got, want)
    assert torch.equal(torch.autograd.grad(got, spec, g)[0], torch.autograd.grad(want, spec, g)[0])
    with torch.no_grad():
        assert torch.equal(mod.stft(x, **kw), mod.stft(x.detach(), **kw)) and not mod.stft(x, **kw).requires_grad
    # what has more to see goes the other way: lazy views, tangents, transforms, a window on the host
    conj = spec.detach().conj()
    assert native._istft_direct(conj, win, 512, 128, 400, 4000, True, False) is None
    assert native._stft_direct(x, win.detach().cpu(), 512, 128, 400, True, False) is None
    assert torch.equal(mod.stft(x, **{**kw, "window": win.detach().cpu()}), mod.stft(x, **kw))
    with pytest.raises(Exception):
        torch.func.jvp(lambda t: mod.stft(t, **kw), (x,), (torch.ones_like(x),))
    with pytest.raises(Exception):
        torch.func.vmap(lambda t: mod.stft(t, **kw))(x.detach().expand(2, *shape))


# Long frames-major signals walk their frames in streams: every frame size that does, hops of a half, a quarter and five
# sixteenths, rows off 8 bytes (odd lengths), edges that fold, missing neighbours, more and fewer samples than the frames cover.
@pytest.mark.gpu
@pytest.mark.parametrize("n_fft,hop,batch,samples,center", [
    (128, 32, 16, 300_001, True), (256, 64, 16, 400_003, True), (256, 80, 5, 1_048_575, False), (512, 128, 16, 400_000, True),
    (512, 256, 3, 2_000_001, True), (2048, 512, 16, 1_000_001, True), (2048, 640, 2, 9_000_000, False),
    (2048, 1024, 8, 2_000_003, True),
])
def test_streamed_inverse_matches_64_bits(n_fft, hop, batch, samples, center):
    torch.manual_seed(0)
    win = torch.hann_window(n_fft - n_fft // 8, device="cuda")
    x = torch.randn(batch, samples, device="cuda", requires_grad=True)
    kw = dict(n_fft=n_fft, hop_length=hop, win_length=win.numel(), window=win, center=center)
    spec = stft(x, **kw)
    g = torch.randn(spec.shape[0], spec.shape[2], spec.shape[1], dtype=torch.complex64, device="cuda").transpose(1, 2)
    (grad,) = torch.autograd.grad(spec, x, g)
    padded = torch.nn.functional.pad(win.double(), (n_fft // 16, n_fft // 16))
    kw64 = dict(n_fft=n_fft, hop_length=hop, window=padded, center=center)
    x64 = x.detach().double().requires_grad_()
    spec64 = torch.stft(x64, pad_mode="reflect", return_complex=True, **kw64)
    (grad64,) = torch.autograd.grad(spec64, x64, g.to(torch.complex128))

    def close(got, want):  # a few roundings of 2^-24 per radix and per frame, against the result's size
        assert (got.double() - want).norm() <= 4e-7 * want.norm() and (got.double() - want).abs().max() <= 4e-6 * want.abs().max()

    close(grad, grad64)
    if not center:
        return
    for length in (samples, samples + 3 * n_fft + 1, samples - 5 * hop - 3):
        got = istft(g, length=length, **kw)
        cover = istft(torch.ones_like(g), length=length, **kw)  # torch refuses what no frame covers
        want = torch.istft(g.to(torch.complex128), length=min(length, samples), **kw64)
        close(got[:, :want.shape[1] - n_fft], want[:, :want.shape[1] - n_fft])
        end = (g.shape[2] - 1) * hop + n_fft // 2
        assert torch.isfinite(got).all() and (length <= end or not got[:, end:].any()) and cover.shape == got.shape


# Streams, one CTA per SM and whole CTAs per signal, only where they leave no more of the device idle than they gain: times of the
# two kernels (B200) differ by 5 % at least in every row.
@pytest.mark.parametrize("n_fft,hop,samples,inverse,streams,batches", [
    (128, 16, 1 << 20, False, (16, 80), ()), (128, 32, 300000, True, (16, 50, 80), ()), (128, 64, 1 << 16, False, (80, 96, 160), ()),
    (256, 64, 1 << 20, False, (8, 16, 24, 32, 50, 64, 96, 120), (80,)),
    (256, 32, 300000, True, (50, 80, 160), ()),
    (256, 128, 1 << 16, True, (120, 148), (50, 80, 96, 160)),
    (512, 128, 1 << 20, True, (8, 16, 24, 32, 64, 120), (80, 96)),
    (512, 128, 300000, False, (32,), (16, 80)),
    (512, 256, 1 << 18, False, (64, 120, 148), (80, 96, 160)),
    (2048, 512, 1 << 20, False, (24, 32, 50, 64, 120), (80, 96)),
    (2048, 512, 1 << 18, True, (120, 148, 160), (50, 80, 96)),
    (2048, 1024, 1 << 18, False, (120, 148, 160), (32, 50, 80, 96)),
    (2048, 1024, 1 << 20, True, (64, 120), (8, 16, 32, 50, 80, 96)),
])
def test_streams_where_they_fill_the_device(n_fft, hop, samples, inverse, streams, batches):
    native = mccl_b200.require_native()
    assert all(native._test_stft_inverse_streams(n_fft, hop, samples, b, inverse) for b in streams)
    assert not any(native._test_stft_inverse_streams(n_fft, hop, samples, b, inverse) for b in batches)


# So many signals that one CTA has all of one, both folded edges too.
@pytest.mark.gpu
@pytest.mark.parametrize("n_fft,hop,batch,samples", [(128, 32, 120, 50_001), (256, 64, 120, 65_537), (512, 256, 148, 100_003),
                                                     (2048, 512, 120, 262_147), (2048, 1024, 120, 524_301)])
def test_streamed_inverse_of_many_signals_matches_64_bits(n_fft, hop, batch, samples):
    native = mccl_b200.require_native()
    assert all(native._test_stft_inverse_streams(n_fft, hop, samples, batch, inverse) for inverse in (False, True))
    test_streamed_inverse_matches_64_bits(n_fft, hop, batch, samples, True)


# Rounding errors of the forward transform and of the inverse's gradient, 2-norm against 64 bits, as the butterflies have them that
# round a turn by an eighth and the sum after it once (times 1e8, the same within 0.1 % for any noise).  With a rounding of its own
# for the turn they are 1.2 to 2.3 % larger.
@pytest.mark.gpu
@pytest.mark.parametrize("n_fft,forward,inverse_gradient", [(128, 9.429, 10.508), (256, 10.117, 11.067), (512, 10.834, 11.735),
                                                            (1024, 11.515, 12.400), (2048, 12.260, 13.061), (4096, 12.831, 13.626)])
def test_packed_butterflies_round_as_scalar_ones(n_fft, forward, inverse_gradient):
    gen = torch.Generator().manual_seed(n_fft)
    samples, hop = 1 << 18, n_fft // 4
    win = torch.hann_window(n_fft, device="cuda")
    x = (0.3 * torch.randn(8, samples, generator=gen)).cuda()
    spec = torch.randn(8, 1 + samples // hop, n_fft // 2 + 1, dtype=torch.complex64, generator=gen).cuda().transpose(1, 2)
    kw, kw64 = dict(n_fft=n_fft, hop_length=hop, win_length=n_fft), dict(n_fft=n_fft, hop_length=hop, window=win.double())
    got = stft(x, window=win, **kw)
    want = torch.stft(x.double(), pad_mode="reflect", return_complex=True, **kw64)
    assert (got - want).norm() <= 1.005e-8 * forward * want.norm()
    spec.requires_grad_()
    (got,) = torch.autograd.grad(istft(spec, window=win, length=samples, **kw), spec, x)
    spec64 = spec.detach().to(torch.complex128).requires_grad_()
    (want,) = torch.autograd.grad(torch.istft(spec64, length=samples, **kw64), spec64, x.double())
    assert (got - want).norm() <= 1.005e-8 * inverse_gradient * want.norm()
