"""The split step of 256 x 256 planes (step_split.cuh) at the x extents that test_gpu_step_kernels.py
leaves out: FP64 has another block of columns, thread count and shared-memory stride than FP32, and
nx = 256 is the widest x part (1024 threads, radix 16 x 16).  Reference and tolerances: as there."""
import pytest

from test_gpu_step_kernels import _compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,precision", [(nx, p) for nx in (8, 32, 64, 256) for p in ("fp64", "mixed")]
                         + [(nx, "fp64") for nx in (48, 96, 128)])
def test_split_step_x_extents(gpu, nx, precision):
    _compare((nx, 256, 256), precision, [3, 11], 0)
