"""Fused AdamW kernel vs torch.optim.AdamW, and per-bucket stepping inside backward (one GPU)."""
import copy

import pytest
import torch

from mccl_b200.utils.spawn import run_workers

pytestmark = pytest.mark.gpu


def test_fused_adamw_matches_torch(cuda_device):
    from mccl_b200.optim import FusedAdamW
    torch.manual_seed(0)
    shapes = [(1000, 333), (333,), (7,), (64, 64, 3), (100003,)]
    p1 = [torch.randn(s, device=cuda_device, requires_grad=True) for s in shapes]
    p2 = [p.detach().clone().requires_grad_(True) for p in p1]
    o1 = FusedAdamW(p1, lr=1e-2, weight_decay=0.05)
    o2 = torch.optim.AdamW(p2, lr=1e-2, weight_decay=0.05)
    for step in range(5):
        for a, b in zip(p1, p2):
            g = torch.randn_like(a)
            a.grad = g.clone(); b.grad = g.clone()
        o1.step(); o2.step()
    for a, b in zip(p1, p2):
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-6), (a - b).abs().max()
    # interchangeable state
    o2.load_state_dict(o1.state_dict())
    o1.load_state_dict(o2.state_dict())


def test_step_follows_what_changes_between_steps(cuda_device):
    # Everything that takes a step off the one-call path and back: a missing gradient, a moved or non-contiguous one, a
    # replaced parameter, counters loaded from a checkpoint, changed hyper-parameters.
    from mccl_b200.optim import FusedAdamW
    torch.manual_seed(1)
    shapes = [(64, 32), (32,), (5000,)]
    p1 = [torch.nn.Parameter(torch.randn(s, device=cuda_device)) for s in shapes]
    p2 = [torch.nn.Parameter(p.detach().clone()) for p in p1]
    o1, o2 = FusedAdamW(p1, lr=1e-2), torch.optim.AdamW(p2, lr=1e-2)

    def step(change=None):
        for i, (a, b) in enumerate(zip(p1, p2)):
            g = torch.randn_like(a)
            a.grad, b.grad = g.clone(), g.clone()
            if change == "missing" and i == 1:
                a.grad = b.grad = None
            if change == "strided" and i == 0:
                a.grad = g.t().contiguous().t()
        o1.step()
        o2.step()
        for a, b in zip(p1, p2):
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-6), change
            sa, sb = o1.state[a], o2.state[b]
            assert float(sa["step"]) == float(sb["step"]) and torch.allclose(sa["exp_avg"], sb["exp_avg"], atol=1e-6)

    step()
    step()
    step("strided")
    step()
    for o in (o1, o2):
        o.param_groups[0]["lr"] = 3e-3
        o.param_groups[0]["weight_decay"] = 0.1
    step()
    o1.load_state_dict(copy.deepcopy(o2.state_dict()))  # (without the copy the two would share their moments)
    step()
    with torch.no_grad():
        p1[0].data = p1[0].detach().clone()  # another address
    step()
    for a, b in zip(p1, p2):
        a.grad = b.grad = None
    before = [p.detach().clone() for p in p1]
    o1.step()
    assert all(torch.equal(p, q) for p, q in zip(p1, before))
    assert o1.state[p1[0]]["step"] == o2.state[p2[0]]["step"]
    step("missing")
    step()  # the counters differ from here on: every parameter has its own bias correction
    step("strided")
    step()


@pytest.mark.parametrize("fused_checkpoint", [False, True])
def test_checkpoint_with_unequal_step_counters(cuda_device, fused_checkpoint):
    # A parameter that joined late, early in training, where the bias corrections differ most.  torch's fused optimizer
    # keeps its counters on the device, and so does its checkpoint.
    from mccl_b200.optim import FusedAdamW
    torch.manual_seed(2)
    shapes = [(100,), (33, 7), (4097,)]
    p1 = [torch.nn.Parameter(torch.randn(s, device=cuda_device)) for s in shapes]
    p2 = [torch.nn.Parameter(p.detach().clone()) for p in p1]
    o1 = FusedAdamW(p1, lr=1e-2)
    o2 = torch.optim.AdamW(p2, lr=1e-2, fused=fused_checkpoint)
    for i in range(6):
        for j, (a, b) in enumerate(zip(p1, p2)):
            g = None if i < 2 and j == 1 else torch.randn_like(b)
            b.grad = g
            a.grad = None if g is None else g.clone()
        o2.step()
        if i < 2:
            for a, b in zip(p1, p2):
                a.data.copy_(b.data)
            o1.load_state_dict(copy.deepcopy(o2.state_dict()))
        else:
            o1.step()
        for a, b in zip(p1, p2):
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-6)
            if b in o2.state:
                assert float(o1.state[a]["step"]) == float(o2.state[b]["step"])


def _oib_single(rank, ws):
    import torch
    from mccl_b200.parallel import wrap_ddp
    from mccl_b200.optim import FusedAdamW
    def make():
        torch.manual_seed(3)
        return torch.nn.Sequential(torch.nn.Linear(128, 512), torch.nn.GELU(), torch.nn.Linear(512, 8)).to(device)
    a, b = make(), make()
    oa, ob = FusedAdamW(a.parameters(), lr=1e-3), FusedAdamW(b.parameters(), lr=1e-3)
    da = wrap_ddp(a, device_ids=[device.index], bucket_cap_mb=1)
    db = wrap_ddp(b, device_ids=[device.index], bucket_cap_mb=1, optimizer_in_backward=ob)
    for i in range(4):
        x = torch.randn(8, 128, device=device); y = torch.randint(0, 8, (8,), device=device)
        for d, o in ((da, oa), (db, ob)):
            o.zero_grad(); torch.nn.functional.cross_entropy(d(x), y).backward(); o.step()
    for p, q in zip(a.parameters(), b.parameters()):
        assert torch.equal(p, q)


def test_optimizer_in_backward_world_size_one():
    run_workers(_oib_single, 1, device="cuda", timeout=180)


def _oib_groups_single(rank, ws):
    import torch
    from mccl_b200.parallel import wrap_ddp
    from mccl_b200.optim import FusedAdamW
    def make():
        torch.manual_seed(5)
        return torch.nn.Sequential(torch.nn.Linear(128, 512), torch.nn.GELU(), torch.nn.Linear(512, 8)).to(device)
    def groups(m):
        return [{"params": [p for p in m.parameters() if p.ndim > 1], "weight_decay": 0.2},
                {"params": [p for p in m.parameters() if p.ndim <= 1], "weight_decay": 0.0, "lr": 5e-3}]
    a, b = make(), make()
    oa, ob = torch.optim.AdamW(groups(a), lr=1e-3), FusedAdamW(groups(b), lr=1e-3)
    sa = torch.optim.lr_scheduler.StepLR(oa, step_size=1, gamma=0.7)
    sb = torch.optim.lr_scheduler.StepLR(ob, step_size=1, gamma=0.7)
    da = wrap_ddp(a, device_ids=[device.index], bucket_cap_mb=25)   # one bucket holding both groups
    db = wrap_ddp(b, device_ids=[device.index], bucket_cap_mb=25, optimizer_in_backward=ob)
    for i in range(5):
        x = torch.randn(8, 128, device=device); y = torch.randint(0, 8, (8,), device=device)
        for d, o, s in ((da, oa, sa), (db, ob, sb)):
            o.zero_grad(); torch.nn.functional.cross_entropy(d(x), y).backward(); o.step(); s.step()
    for p, q in zip(a.parameters(), b.parameters()):
        assert torch.allclose(p, q, rtol=1e-4, atol=2e-5), (p - q).abs().max()
    # a group added later is indexed too
    extra = torch.nn.Parameter(torch.zeros(16, device=device))
    ob.add_param_group({"params": [extra]})
    assert extra.data_ptr() in ob._by_ptr


@pytest.mark.parametrize("python_hook", ["0", "1"])
def test_bucket_spanning_two_param_groups_uses_each_groups_hyperparameters(python_hook):
    run_workers(_oib_groups_single, 1, device="cuda", timeout=180, env={"MCCL_PYTHON_BUCKET_HOOK": python_hook})


def _oib_unequal_single(rank, ws):
    import copy

    import torch
    from mccl_b200.parallel import wrap_ddp
    from mccl_b200.optim import FusedAdamW
    def make():
        torch.manual_seed(7)
        return torch.nn.Sequential(torch.nn.Linear(128, 512), torch.nn.GELU(), torch.nn.Linear(512, 8)).to(device)
    a, b = make(), make()
    for m in (a, b):
        m[0].bias.requires_grad_(False)
    order = lambda m: [m[0].bias, m[2].weight, m[2].bias, m[0].weight]  # a frozen parameter comes first
    oa, ob = torch.optim.AdamW(order(a), lr=1e-2), FusedAdamW(order(b), lr=1e-2)
    x = torch.randn(8, 128, device=device); y = torch.randint(0, 8, (8,), device=device)
    torch.nn.functional.cross_entropy(a(x), y).backward()
    a[0].weight.grad = None                     # first steps without this one
    for _ in range(2):
        oa.step()
    b.load_state_dict(a.state_dict())
    db = wrap_ddp(b, device_ids=[device.index], bucket_cap_mb=25, optimizer_in_backward=ob)
    ob.load_state_dict(copy.deepcopy(oa.state_dict()))
    for i in range(5):
        x = torch.randn(8, 128, device=device); y = torch.randint(0, 8, (8,), device=device)
        for d, o in ((a, oa), (db, ob)):
            o.zero_grad(); torch.nn.functional.cross_entropy(d(x), y).backward(); o.step()
    for p, q in zip(order(a), order(b)):
        assert torch.allclose(p, q, rtol=1e-4, atol=2e-5), (p - q).abs().max()
        if p.requires_grad:
            assert float(oa.state[p]["step"]) == float(ob.state[q]["step"])


@pytest.mark.parametrize("python_hook", ["0", "1"])
def test_optimizer_in_backward_with_unequal_step_counters(python_hook):
    run_workers(_oib_unequal_single, 1, device="cuda", timeout=180, env={"MCCL_PYTHON_BUCKET_HOOK": python_hook})
