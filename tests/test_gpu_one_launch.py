"""One-launch sweeps (sweep_cluster.cuh): what the comparisons with the step passes in
test_gpu_step_kernels.py do not show."""
import numpy as np
import pytest

from polyswift_plusplus_b200.scft import ScftSolver
from test_gpu_step_kernels import _case

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 24, 32, 48, 64, 96, 128])
def test_mixed_films_repeat_bit_for_bit(gpu, n):
    """The mean-mode sums of a step reach every CTA before those of the next: from the same
    fields, every run gives the same bits."""
    cfg, w = _case((n, n, 1), "mixed", 60)
    s = ScftSolver(cfg)
    s.set_variant(3)
    first = None
    for _ in range(12):
        s.restore(w)
        s.update(2)
        got = [s.w(0), s.w(1), s.phi(0), s.phi(1)]
        first = first or got
        assert all(np.array_equal(a, b) for a, b in zip(got, first))
    s.close()


@pytest.mark.parametrize("n,precision", [((32, 32, 32), "fp64"), ((24, 24, 24), "fp64"), ((128, 128, 1), "fp64"),
                                         ((128, 128, 1), "mixed"), ((8, 8, 8), "mixed")])
def test_wait_timeout_of_a_long_sweep(gpu, n, precision):
    """With a poll limit of 0 every CTA's first wait gives up, and the CTAs stop sending: a sweep
    whose later steps would have sent the barriers more than 2^20 bytes ends, is reported, and a
    new handle's run is the undisturbed one's."""
    from polyswift_plusplus_b200 import _abi as A
    cfg, w = _case(n, precision, 200)
    s = ScftSolver(cfg)
    s.set_variant(3)
    s.restore(w)
    s.update(2)
    want = [s.w(0), s.phi(1)]
    for _ in range(3):
        s.restore(w)
        assert gpu.ps_gpu_set_bulk_wait_limit(0) == A.PS_OK
        try:
            with pytest.raises(A.PsError) as ei:
                s.update(1)
        finally:
            assert gpu.ps_gpu_set_bulk_wait_limit(0xFFFFFFFF) == A.PS_OK
        assert ei.value.code == A.PS_GPU_ERR and "wait limit" in str(ei.value)
    s.close()
    s = ScftSolver(cfg)
    s.set_variant(3)
    s.restore(w)
    s.update(2)
    assert all(np.array_equal(a, b) for a, b in zip(want, [s.w(0), s.phi(1)]))
    s.close()


def test_adjoint_after_a_wait_timeout(gpu):
    """A backward pass that timed out leaves the forward pass valid: the next backward pass gives
    the undisturbed gradients.  A forward pass that timed out leaves none."""
    import torch
    from polyswift_plusplus_b200 import _abi as A
    from polyswift_plusplus_b200 import workloads as W
    from polyswift_plusplus_b200.adjoint import ChainAdjoint
    cfg = W.diblock_config(16, 2.0, 0.35, 20.0, 20, W.Updater(kind="steepestDescent"), "fp64")
    g = torch.Generator(device="cuda").manual_seed(3)
    w = torch.rand((2, cfg.n_total), generator=g, dtype=torch.float64, device="cuda")

    def timed_out(call):
        assert gpu.ps_gpu_set_bulk_wait_limit(0) == A.PS_OK
        try:
            with pytest.raises(A.PsError) as ei:
                call()
        finally:
            assert gpu.ps_gpu_set_bulk_wait_limit(0xFFFFFFFF) == A.PS_OK
        assert ei.value.code == A.PS_GPU_ERR and "wait limit" in str(ei.value)

    with_gphi = torch.ones_like(w)
    adj = ChainAdjoint(cfg)
    adj.forward(w)
    want = adj.backward(with_gphi, 0.5)[0].clone()
    timed_out(lambda: adj.backward(with_gphi, 0.5))
    assert torch.equal(adj.backward(with_gphi, 0.5)[0], want)
    timed_out(lambda: adj.forward(w))
    with pytest.raises(A.PsError) as ei:
        adj.backward(with_gphi, 0.5)
    assert ei.value.code == A.PS_ATTRIB_ERR
    adj.forward(w)
    assert torch.equal(adj.backward(with_gphi, 0.5)[0], want)
    adj.close()


def test_one_launch_grids_of_this_device(gpu):
    """The whole device has room for every cluster; other grids have no such kernel."""
    import ctypes as C
    from polyswift_plusplus_b200 import _abi as A
    from test_gpu_step_kernels import ONE_LAUNCH
    for precision in (A.PS_PREC_FP64, A.PS_PREC_MIXED):
        for n in ONE_LAUNCH:
            assert gpu.ps_gpu_one_launch((C.c_int * 3)(*n), precision) == 1, n
        for n in ((48, 48, 48), (16, 16, 24), (128, 64, 1), (20, 20, 20)):
            assert gpu.ps_gpu_one_launch((C.c_int * 3)(*n), precision) == 0, n


TUNE = """
import sys
sys.path[:0] = {paths}
from test_gpu_step_kernels import _case
from polyswift_plusplus_b200.scft import ScftSolver
cfg, w = _case((24, 48, 48), "fp64", 100)
for _ in range(3):
    s = ScftSolver(cfg)
    s.restore(w)
    s.update(2)
    print(*s.variant()[1])
    s.close()
"""


def test_tuner_times_no_kernel_loading(gpu):
    """The times of a fresh process's first handle are those of the next ones: a pass takes about
    1 ms here, loading the kernels of a variant about 20."""
    import subprocess
    import sys
    from pathlib import Path
    here = Path(__file__).resolve().parent
    out = subprocess.run([sys.executable, "-c", TUNE.format(paths=[str(here.parent), str(here)])], check=True,
                         capture_output=True, text=True).stdout
    first, *later = [[float(x) for x in line.split()] for line in out.splitlines()]
    for v, ms in enumerate(first):
        assert ms <= 2 * min(t[v] for t in later) + 2.0 or ms < 0, (v, ms)
    assert sum(ms > 0 for ms in first) == 8


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", [16, 24, 32, 48, 64, 96, 128])
def test_one_row_planes(gpu, n, precision):
    """n x 1 x n grids take the films' one-launch sweeps with the tables of another axis."""
    from test_gpu_step_kernels import _compare
    _compare((n, 1, n), precision, [3, 11], 0)


@pytest.mark.parametrize("n", [(24, 24, 1), (64, 64, 1), (128, 128, 1), (32, 1, 32), (12, 12, 12)])
def test_adjoint_on_one_launch_grids(gpu, n):
    """Forward and recomputation in one launch each, the adjoint steps in separate passes."""
    from test_gpu_adjoint_steps import test_adjoint_schedules
    test_adjoint_schedules(gpu, n)
