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
