"""The fused adjoint steps (square y-z planes of extents 16 to 128) at every plane size, against
torch's own differentiation of the same discrete forward in FP64.  Tolerance: both sides are exact
derivatives of the same sums; about 100 roundings of 1e-16 on each term, below 1e-10 of the
gradient's maximum."""
import dataclasses
import math

import numpy as np
import pytest
import torch

from polyswift_plusplus_b200 import workloads as W
from polyswift_plusplus_b200.adjoint import ChainAdjoint

pytestmark = pytest.mark.gpu


def _weights(steps):
    c = [0.0] * (steps + 1)
    num = steps + 1
    for n in range(0, num - 3 if num % 2 == 0 else num - 2, 2):
        c[n] += 0.33333
        c[n + 1] += 4 * 0.33333
        c[n + 2] += 0.33333
    if num % 2 == 0:
        c[-2] += 0.5
        c[-1] += 0.5
    return c


def _torch_forward(cfg, w, box, ds):
    grid, steps = cfg.n, [b for b in (7, 13)]
    k2 = 0.0
    for d in range(3):
        i = torch.fft.fftfreq(grid[d], dtype=torch.float64, device="cuda") * grid[d]
        if d == 2:
            i = i[: grid[d] // 2 + 1]
        k = 2 * math.pi * i.abs() / box[d].to("cuda")
        k2 = k2 + (k * k).reshape([-1 if a == d else 1 for a in range(3)])
    d2 = ds.to("cuda")

    def sweep(q, b):
        e, g = torch.exp(-0.5 * d2[b] * w[b].reshape(grid)), torch.exp(-d2[b] * k2)
        out = [q]
        for _ in range(steps[b]):
            q = e * torch.fft.irfftn(g * torch.fft.rfftn(e * q), s=grid)
            out.append(q)
        return out
    one = torch.ones(grid, dtype=torch.float64, device="cuda")
    a0 = sweep(one, 0)
    a1 = sweep(a0[-1], 1)
    b1 = sweep(one, 1)
    b0 = sweep(b1[-1], 0)
    q = (a0[0] * b0[-1]).mean()
    phi = []
    for b, (f, r) in enumerate(((a0, b0), (a1, b1))):
        c = _weights(steps[b])
        phi.append(sum(c[n] * f[n] * r[steps[b] - n] for n in range(steps[b] + 1)) * d2[b] / q)
    return torch.stack(phi).reshape(2, -1), torch.log(q)


@pytest.mark.parametrize("m", [16, 24, 32, 48, 64, 96, 128])
def test_fused_adjoint_steps(gpu, m):
    cfg = W.diblock_config(16, 2.0, 0.35, 20.0, 20, W.Updater(kind="steepestDescent"), "fp64")
    cfg = dataclasses.replace(cfg, n=(4, m, m), cell=(0.13, 0.07, 0.06))
    rng = np.random.default_rng(m)
    w = torch.tensor(rng.uniform(-1, 1, (2, cfg.n_total)), device="cuda")
    gphi = torch.tensor(rng.standard_normal((2, cfg.n_total)), device="cuda")
    for checkpoint in (0, 1):
        adj = ChainAdjoint(cfg, checkpoint=checkpoint)
        phi, lnq = adj.forward(w)
        gw, gbox, gds = adj.backward(gphi, 0.7)
        wt = w.clone().requires_grad_(True)
        box = torch.tensor([cfg.n[d] * cfg.cell[d] for d in range(3)], dtype=torch.float64, requires_grad=True)
        ds = torch.full((2,), 1.0 / 20, dtype=torch.float64, requires_grad=True)
        tphi, tlnq = _torch_forward(cfg, wt, box, ds)
        ((tphi * gphi).sum() + 0.7 * tlnq).backward()
        assert abs(lnq - tlnq.item()) < 1e-12
        for got, ref in ((phi, tphi.detach()), (gw, wt.grad), (torch.tensor(gbox), box.grad), (torch.tensor(gds), ds.grad)):
            assert (got - ref).abs().max().item() <= 1e-10 * ref.abs().max().item(), (m, checkpoint)
        adj.close()


@pytest.mark.parametrize("n", [(16, 16, 16), (48, 48, 48), (24, 32, 32), (128, 16, 16)])
def test_adjoint_schedules(gpu, n):
    """One-launch and stepwise sweeps, both adjoints together (nx <= 96) and one at a time: the
    results do not depend on the checkpoint interval (whole, uneven and single segments), bit for
    bit, and match torch."""
    cfg = W.diblock_config(16, 2.0, 0.35, 20.0, 20, W.Updater(kind="steepestDescent"), "fp64")
    cfg = dataclasses.replace(cfg, n=n, cell=(0.08, 0.07, 0.06))
    rng = np.random.default_rng(sum(n))
    w = torch.tensor(rng.uniform(-1, 1, (2, cfg.n_total)), device="cuda")
    gphi = torch.tensor(rng.standard_normal((2, cfg.n_total)), device="cuda")
    wt = w.clone().requires_grad_(True)
    box = torch.tensor([cfg.n[d] * cfg.cell[d] for d in range(3)], dtype=torch.float64, requires_grad=True)
    ds = torch.full((2,), 1.0 / 20, dtype=torch.float64, requires_grad=True)
    tphi, tlnq = _torch_forward(cfg, wt, box, ds)
    ((tphi * gphi).sum() + 0.7 * tlnq).backward()
    first = None
    for checkpoint in (1, 0, 7, 20):
        adj = ChainAdjoint(cfg, checkpoint=checkpoint)
        for again in range(2):
            phi, lnq = adj.forward(w)
            gw, gbox, gds = adj.backward(gphi, 0.7)
            got = [phi, torch.tensor([lnq], dtype=torch.float64), gw, torch.tensor(gbox), torch.tensor(gds)]
            if first is None:
                first = got
            assert all(torch.equal(a, b) for a, b in zip(got, first)), (n, checkpoint, again)
        adj.close()
    for got, ref in zip(first, (tphi.detach(), tlnq.detach().cpu().reshape(1), wt.grad, box.grad, ds.grad)):
        assert (got - ref).abs().max().item() <= 1e-10 * max(ref.abs().max().item(), 1e-2), n


def test_adjoint_wait_timeout_is_reported(gpu):
    """With a poll limit of 0 the one-launch sweeps' waits give up: forward and backward report it."""
    from polyswift_plusplus_b200 import _abi as A
    cfg = W.diblock_config(16, 2.0, 0.35, 20.0, 20, W.Updater(kind="steepestDescent"), "fp64")
    w = torch.zeros((2, cfg.n_total), dtype=torch.float64, device="cuda")
    adj = ChainAdjoint(cfg)
    for step in ("forward", "backward"):
        if step == "backward":
            ref, _ = adj.forward(w)
        assert gpu.ps_gpu_set_bulk_wait_limit(0) == A.PS_OK
        try:
            with pytest.raises(A.PsError) as ei:
                adj.forward(w) if step == "forward" else adj.backward(torch.ones_like(w), 1.0)
        finally:
            assert gpu.ps_gpu_set_bulk_wait_limit(0xFFFFFFFF) == A.PS_OK
        assert ei.value.code == A.PS_GPU_ERR and "wait limit" in str(ei.value)
    phi, _ = adj.forward(w)
    assert torch.equal(phi, ref)
    adj.close()
