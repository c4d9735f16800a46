"""Top-k compression kernels vs the host TopKCompressor (the oracle)."""
import struct

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _oracle_pairs(native, adjusted_source, ratio, stable_id=0, comp=None):
    comp = comp or native.TopKCompressor(ratio)
    blob = comp.compress(adjusted_source.cpu().float().contiguous(), stable_id)
    k = struct.unpack_from("<I", blob, 0)[0]
    rec = np.frombuffer(blob, dtype=np.dtype([("i", "<u4"), ("v", "<f4")]), offset=4, count=k)
    return comp, rec["i"].astype(np.int64).tolist(), rec["v"].tolist()


@pytest.mark.parametrize("n,ratio", [(10, 0.5), (1000, 0.01), (65537, 0.1), (1_000_003, 0.01), (300_001, 1.0)])
def test_select_matches_host_oracle(native, cuda_device, n, ratio):
    g = torch.randn(n)
    comp, idx, val = _oracle_pairs(native, g, ratio)
    res = torch.zeros(n, device=cuda_device)
    pairs = native._topk_select(g.to(cuda_device), res, ratio)
    torch.cuda.synchronize()
    got_idx = pairs[:, 0].cpu().tolist()
    got_val = pairs[:, 1].cpu().view(torch.float32).tolist()
    assert got_idx == idx
    assert got_val == val
    assert torch.equal(res.cpu(), comp.residual(0))


def test_select_ties_take_lower_index(native, cuda_device):
    g = torch.tensor([1.0, -2.0, 2.0, 2.0, -2.0, 0.5, 2.0, 3.0])
    res = torch.zeros(8, device=cuda_device)
    pairs = native._topk_select(g.to(cuda_device), res, 0.5)  # k = 4: 3.0 and three of the |2.0|
    assert pairs[:, 0].cpu().tolist() == [1, 2, 3, 7]
    assert res.cpu().tolist() == [1.0, 0.0, 0.0, 0.0, -2.0, 0.5, 2.0, 0.0]


@pytest.mark.parametrize("kind", ["few_magnitudes", "mostly_zero", "all_equal", "bf16_grid"])
def test_select_on_heavily_tied_data_matches_host_oracle(native, cuda_device, kind):
    # Many elements share the k-th magnitude (or it is zero): threshold and ties come from the whole
    # vector, and the ties must still go to the lowest indices, exactly like the host implementation.
    n, ratio = 400_003, 0.02
    gen = torch.Generator().manual_seed(11)
    if kind == "few_magnitudes":
        g = torch.randint(-3, 4, (n,), generator=gen).float()
    elif kind == "mostly_zero":
        g = torch.zeros(n)
        nz = torch.randperm(n, generator=gen)[: n // 500]
        g[nz] = torch.randn(n // 500, generator=gen)
    elif kind == "all_equal":
        g = torch.full((n,), -0.75)
    else:
        g = torch.randn(n, generator=gen).bfloat16().float().mul(8).round().div(8)   # coarse grid: many exact ties
    comp, idx, val = _oracle_pairs(native, g, ratio)
    res = torch.zeros(n, device=cuda_device)
    pairs = native._topk_select(g.to(cuda_device), res, ratio)
    torch.cuda.synchronize()
    assert pairs[:, 0].cpu().tolist() == idx
    assert pairs[:, 1].cpu().view(torch.float32).tolist() == val
    assert torch.equal(res.cpu(), comp.residual(0))
    # a second call on the same residual (now with holes where entries were sent) stays exact too
    _, idx2, _ = _oracle_pairs(native, g, ratio, comp=comp)
    pairs2 = native._topk_select(g.to(cuda_device), res, ratio)
    assert pairs2[:, 0].cpu().tolist() == idx2
    assert torch.equal(res.cpu(), comp.residual(0))


def test_error_feedback_accumulates_like_oracle(native, cuda_device):
    n, ratio = 50_000, 0.02
    comp = native.TopKCompressor(ratio)
    res = torch.zeros(n, device=cuda_device)
    for step in range(5):
        g = torch.randn(n, generator=torch.Generator().manual_seed(step))
        _, idx, val = _oracle_pairs(native, g, ratio, comp=comp)
        pairs = native._topk_select(g.to(cuda_device), res, ratio)
        assert pairs[:, 0].cpu().tolist() == idx, f"step {step}"
        assert torch.equal(res.cpu(), comp.residual(0))


@pytest.mark.parametrize("ws", [2, 4, 8])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_fused_topk_allreduce_is_consistent(native, cuda_device, ws, dtype):
    n, ratio = 200_003, 0.01
    grp = native.EmuGroup(ws, 8 << 20)
    grads = [torch.randn(n, generator=torch.Generator().manual_seed(r)).to(dtype).to(cuda_device) for r in range(ws)]
    orig = [g.clone() for g in grads]
    residuals = [torch.zeros(n, device=cuda_device) for _ in range(ws)]
    grp.topk_allreduce(grads, residuals, ratio, 1.0 / ws)
    torch.cuda.synchronize()
    for r in range(1, ws):
        assert torch.equal(grads[0], grads[r]), "dense results differ across ranks"
    # dense reference: sum over ranks (in rank order) of each rank's sparse selection, scaled
    dense = torch.zeros(n, dtype=torch.float32)
    scale = torch.tensor(1.0 / ws, dtype=torch.float32)
    for r in range(ws):
        comp, idx, val = _oracle_pairs(native, orig[r].float(), ratio)
        if dtype == torch.float32:
            dense[idx] += torch.tensor(val) * scale
        else:
            dense[idx] = (dense[idx].to(dtype).float() + torch.tensor(val) * scale).to(dtype).float()
        assert torch.equal(residuals[r].cpu(), comp.residual(0))
    assert torch.equal(grads[0].float().cpu(), dense.to(dtype).float())


def _data(kind, n, dtype):
    gen = torch.Generator().manual_seed(n)
    g = 1e-3 * torch.randn(n, generator=gen)
    r = 2e-3 * torch.randn(n, generator=gen)
    if kind == "grid":            # 16-bit values and no residual yet: ties at every magnitude
        g, r = g.bfloat16().float(), torch.zeros(n)
    elif kind == "sparse":        # fewer non-zeros than entries to send: zeros are sent, lowest index first
        g, r = torch.zeros(n), torch.zeros(n)
        g[torch.randperm(n, generator=gen)[: max(1, n // 300)]] = 1.0
    elif kind == "rows":          # an embedding's gradient: whole rows, the rest zero
        g, r = g * (torch.rand(n // 1024 + 1, generator=gen) < 0.05).float().repeat_interleave(1024)[:n], torch.zeros(n)
    elif kind == "levels":        # far more ties at the threshold than a candidate list holds
        g, r = torch.randint(-3, 4, (n,), generator=gen).float(), torch.zeros(n)
    elif kind == "steps":         # a crowded bin, within what the list holds or not
        g, r = (8 * torch.randn(n, generator=gen)).round(), torch.zeros(n)
    elif kind == "wide":          # magnitudes over the whole range of the type, infinities among them
        r = torch.zeros(n)
        g = torch.ldexp(1 + torch.rand(n, generator=gen), torch.randint(-140, 127, (n,), generator=gen))
        g[:: n // 3] = float("inf")
    return g.to(dtype), r


# One cluster launch up to 8 x 48 Ki elements, sample + adjust + select + output above; sizes around that limit, around the tile of
# 1024 and the group of tiles, odd sizes, and every kind of data for which the sampled magnitude misses (fewer than k reach
# it, or more than the list holds).  Integer selection rule: exact.
@pytest.mark.parametrize("n,ratio", [(1, 1.0), (7, 0.5), (393_216, 0.01), (393_217, 0.01), (786_432, 0.1), (786_433, 0.01),
                                     (1_048_577, 0.001), (3_000_001, 0.1), (9_437_184, 0.01), (2_000_000, 1.0)])
@pytest.mark.parametrize("kind", ["normal", "grid", "sparse", "rows", "levels", "steps", "wide"])
def test_select_and_dense_paths_match_host_oracle(native, cuda_device, one_rank, n, ratio, kind):
    if n < 100 and kind != "normal":
        pytest.skip("the kinds differ for many elements only")
    dtype = torch.bfloat16 if n % 2 == 0 and kind != "wide" else torch.float32
    g, r = _data(kind, n, dtype)
    adjusted = g.float() + r
    comp, idx, val = _oracle_pairs(native, adjusted, ratio)
    idx, val = torch.tensor(idx), torch.tensor(val)
    # pairs
    res = r.to(cuda_device)
    grad = g.to(cuda_device)
    pairs = native._topk_select(grad, res, ratio).cpu()
    assert torch.equal(pairs[:, 0].long(), idx)
    assert torch.equal(pairs[:, 1].view(torch.float32), val)
    assert torch.equal(res.cpu(), comp.residual(0))
    assert torch.equal(grad.cpu(), g)
    # dense, from arrays that are not 16-byte aligned
    res = torch.zeros(n + 1, device=cuda_device)[1:]
    grad = torch.zeros(n + 1, device=cuda_device, dtype=dtype)[1:]
    res.copy_(r)
    grad.copy_(g)
    one_rank.allreduce_topk(grad, res, ratio, 0.25).wait()
    want = torch.zeros(n)
    want[idx] = val * 0.25
    assert torch.equal(grad.cpu(), want.to(dtype))
    assert torch.equal(res.cpu(), comp.residual(0))


# k at the end of a run of equal magnitudes, where the radix select stops early, one before and one behind; the runs differ in
# the first, the second and the third digit, and the last one is zeros.  Exact.
@pytest.mark.parametrize("k", [99, 100, 101, 250, 299, 300, 301, 600, 601, 999, 1000])
@pytest.mark.parametrize("n", [1000, 20_000])
def test_selection_at_the_end_of_a_run(native, cuda_device, one_rank, n, k):
    gen = torch.Generator().manual_seed(k)
    g = torch.zeros(n)
    g[:1000] = torch.tensor([8.0] * 100 + [1.0 + 2.0 ** -11] * 200 + [1.0 + 2.0 ** -22] * 300 + [0.0] * 400)
    g = torch.where(torch.rand(n, generator=gen) < 0.5, -g, g)[torch.randperm(n, generator=gen)]
    ratio = k / n
    comp, idx, val = _oracle_pairs(native, g, ratio)
    assert len(idx) == k
    res = torch.zeros(n, device=cuda_device)
    pairs = native._topk_select(g.to(cuda_device), res, ratio).cpu()
    assert torch.equal(pairs[:, 0].long(), torch.tensor(idx))
    assert torch.equal(res.cpu(), comp.residual(0))
    grad, res = g.to(cuda_device), torch.zeros(n, device=cuda_device)
    one_rank.allreduce_topk(grad, res, ratio, 0.5).wait()
    want = torch.zeros(n)
    want[torch.tensor(idx)] = torch.tensor(val) * 0.5
    assert torch.equal(grad.cpu(), want) and torch.equal(res.cpu(), comp.residual(0))


def _missing(kind, n, ratio):
    """Data for which the k-th element lies outside what the sampled magnitude bounds."""
    gen = torch.Generator().manual_seed(n)
    g = torch.randn(n, generator=gen)
    if kind == "nonzeros":        # somewhat more non-zeros than entries to send: the bound is the smallest non-zero
        g = g * (torch.rand(n, generator=gen) < 1.1 * ratio)
    elif kind == "two_scales":    # the larger population ends between rank k and the sampled rank
        g = torch.where(torch.rand(n, generator=gen) < 1.1 * ratio, g.sign() * (100 + g.abs()), 0.1 * g)
    elif kind == "two_levels":    # the same with ties on both sides
        g = torch.where(torch.rand(n, generator=gen) < 1.1 * ratio, 64 * g.sign(), 0.25 * g.sign())
    elif kind == "heavy":         # magnitudes over hundreds of octaves
        g = g * torch.exp2(20 * torch.randn(n, generator=gen))
    return g


# k below and above the sampled rank, close to n, and all of n; tiles and groups cut short.  Exact.
@pytest.mark.parametrize("n,ratio", [(393_217, 0.01), (1_048_577, 0.001), (3_000_001, 0.1), (5_000_000, 1e-5), (700_001, 0.99),
                                     (2_000_001, 1.0)])
@pytest.mark.parametrize("kind", ["nonzeros", "two_scales", "two_levels", "heavy", "normal"])
def test_select_where_the_sampled_bound_misses(native, cuda_device, one_rank, n, ratio, kind):
    g = _missing(kind, n, ratio)
    comp, idx, val = _oracle_pairs(native, g, ratio)
    idx, val = torch.tensor(idx), torch.tensor(val)
    res = torch.zeros(n, device=cuda_device)
    pairs = native._topk_select(g.to(cuda_device), res, ratio).cpu()
    assert torch.equal(pairs[:, 0].long(), idx)
    assert torch.equal(pairs[:, 1].view(torch.float32), val)
    assert torch.equal(res.cpu(), comp.residual(0))
    grad, res = g.to(cuda_device), torch.zeros(n, device=cuda_device)
    one_rank.allreduce_topk(grad, res, ratio, 0.5).wait()
    want = torch.zeros(n)
    want[idx] = val * 0.5
    assert torch.equal(grad.cpu(), want)
    assert torch.equal(res.cpu(), comp.residual(0))


def _misled(kind, n, ratio):
    """Data whose sampled elements are smaller than the rest: more than k elements lie above the magnitude up to which the
    first launch of a dense selection sends on its own."""
    gen = torch.Generator().manual_seed(n)
    if kind == "narrow":          # that magnitude and the k-th element's in one crowded bin; the sample is right
        return 1 + 1e-6 * torch.randn(n, generator=gen)
    s = torch.arange(65536, dtype=torch.int64)
    stride = n // 65536
    sampled = s * stride + ((((s * 2654435761) % 2 ** 32) >> 8) * stride >> 24)
    k = int(n * ratio)
    rest = torch.ones(n, dtype=torch.bool)
    rest[sampled] = False
    rest = rest.nonzero()[:, 0]
    large = rest[torch.randperm(rest.numel(), generator=gen)[: int(1.15 * k)]]
    g = 0.01 * torch.rand(n, generator=gen)
    g[sampled] = 0.001 * torch.rand(65536, generator=gen)
    some = sampled[torch.randperm(65536, generator=gen)[: int(1.5 * 65536 * ratio)]]
    g[some] = 0.6 + 0.3 * torch.rand(some.numel(), generator=gen)
    if kind == "octave":          # the k-th element within the histogram, its bin above that magnitude
        g[large] = 1 + 0.3 * torch.rand(large.numel(), generator=gen)
    elif kind == "far":           # beyond it
        g[large] = 64 + torch.rand(large.numel(), generator=gen)
    elif kind == "ties":
        g[large] = 1.0
    elif kind == "crowded":       # one bin, more entries than one block resolves
        g[large] = 1 + 2.0 ** -23 * torch.randint(0, 5, (large.numel(),), generator=gen)
    elif kind == "overflow":      # more than the list holds
        g[rest] = 1 + torch.rand(rest.numel(), generator=gen)
    return torch.where(torch.rand(n, generator=gen) < 0.5, -g, g)


# What was sent too early is taken back: from the list, at the threshold's ties, where the list overflows.  Exact.
@pytest.mark.parametrize("kind,n,ratio", [("octave", 1_000_003, 0.01), ("octave", 524_288, 0.1), ("far", 1_000_003, 0.01),
                                          ("far", 3_000_000, 0.003), ("ties", 1_000_003, 0.01), ("crowded", 20_000_003, 0.01),
                                          ("overflow", 1_000_003, 0.01), ("overflow", 700_001, 0.1),
                                          ("narrow", 20_000_003, 0.01)])
def test_dense_selection_where_the_upper_bound_misses(native, cuda_device, one_rank, kind, n, ratio):
    g = _misled(kind, n, ratio)
    comp, idx, val = _oracle_pairs(native, g, ratio)
    want = torch.zeros(n)
    want[torch.tensor(idx)] = torch.tensor(val) * 0.5
    grad, res = g.to(cuda_device), torch.zeros(n, device=cuda_device)
    one_rank.allreduce_topk(grad, res, ratio, 0.5).wait()
    assert torch.equal(grad.cpu(), want)
    assert torch.equal(res.cpu(), comp.residual(0))


def test_dense_selections_side_by_side(cuda_device, one_rank):
    # Both lanes at once: a grid that is not resident as a whole selects by one cluster, with what was sent early in the list.
    n, ratio = 4_000_001, 0.01
    gs = [_missing("two_scales", n, ratio).to(cuda_device), _misled("far", n, ratio).to(cuda_device)]

    def run(wait_each):
        grads, res = [g.clone() for g in gs], [torch.zeros_like(g) for g in gs]
        works = []
        for g, r in zip(grads, res):
            works.append(one_rank.allreduce_topk(g, r, ratio, 1.0))
            if wait_each:
                works[-1].wait()
        for w in works:
            w.wait()
        torch.cuda.synchronize()
        return grads + res

    want = run(True)
    for _ in range(10):
        assert all(torch.equal(a, b) for a, b in zip(run(False), want))


def _time_us(fn, reset, runs=5):
    best = float("inf")
    for _ in range(runs):
        reset()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        torch.cuda._sleep(200_000)  # the launches are all queued when the first one runs
        a.record()
        fn()
        b.record()
        torch.cuda.synchronize()
        best = min(best, a.elapsed_time(b) * 1e3)
    return best


@pytest.mark.parametrize("kind,ratio", [("two_scales", 0.01), ("nonzeros", 0.01), ("normal", 1.0)])
def test_a_missed_bound_costs_passes_not_a_single_cluster(native, cuda_device, kind, ratio):
    # Eight passes of the whole GPU at the very most against three; one cluster over the vector takes more than tenfold.
    n = 32_000_000
    res = torch.zeros(n, device=cuda_device)

    def cost(g, ratio):
        return _time_us(lambda: native._topk_select(g, res, ratio), res.zero_)

    plain = cost(_missing("normal", n, 0.01).to(cuda_device), 0.01)
    assert cost(_missing(kind, n, ratio).to(cuda_device), ratio) < 5 * plain


def test_a_missed_bound_on_two_streams_at_once(native, cuda_device):
    # Two grids that each want most of the device: whichever is not resident as a whole falls back and stays exact.
    n, ratio = 4_000_001, 0.01
    gs = [_missing("two_scales", n - i, ratio).to(cuda_device) for i in range(2)]
    want = [native._topk_select(g, torch.zeros_like(g), ratio).clone() for g in gs]
    streams = [torch.cuda.Stream() for _ in gs]
    torch.cuda.synchronize()
    for _ in range(10):
        got = []
        for g, s in zip(gs, streams):
            with torch.cuda.stream(s):
                got.append((native._topk_select(g, torch.zeros_like(g), ratio)))
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("megabytes", [28, 8])
def test_selection_without_room_for_the_list(native, cuda_device, one_rank, megabytes):
    # Above the list's size a device has: what the pairs alone would need, and less.  The same results either way.
    n, ratio = 20_000_001, 0.1
    for kind in ("normal", "two_levels"):
        g = _missing(kind, n, ratio).to(cuda_device)
        want_grad, want_res, res = g.clone(), torch.zeros_like(g), torch.zeros_like(g)
        one_rank.allreduce_topk(want_grad, want_res, ratio, 0.5).wait()
        want_pairs = native._topk_select(g, res, ratio)
        got_grad, got_res = g.clone(), torch.zeros_like(g)
        res2 = torch.zeros_like(g)
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        total = torch.cuda.get_device_properties(cuda_device).total_memory
        torch.cuda.set_per_process_memory_fraction((torch.cuda.memory_reserved() + (megabytes << 20)) / total)
        try:
            one_rank.allreduce_topk(got_grad, got_res, ratio, 0.5).wait()
            pairs = native._topk_select(g, res2, ratio) if megabytes > 16 else None
            torch.cuda.synchronize()
        finally:
            torch.cuda.set_per_process_memory_fraction(1.0)
        assert torch.equal(got_grad, want_grad) and torch.equal(got_res, want_res)
        if pairs is not None:
            assert torch.equal(pairs, want_pairs) and torch.equal(res2, res)


@pytest.fixture(scope="module")
def one_rank(cuda_device):
    import torch.distributed as dist

    import mccl_b200

    created = not dist.is_initialized()
    if created:
        dist.init_process_group("mccl", store=dist.HashStore(), rank=0, world_size=1)
    yield mccl_b200.get_backend(device=cuda_device)
    if created:
        dist.destroy_process_group()
