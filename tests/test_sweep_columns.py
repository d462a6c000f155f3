"""How the one-launch sweeps (sweep_cluster.cuh) share the columns of a plane out over the CTAs
of a cluster, on the host: the layout functions that the kernel uses, compiled by nvcc.

A CTA's bar_b phases stay apart because every CTA owes every other one columns: one that owned
none could still be in step k (its mean-mode sums unread) while the sums of step k + 1 arrive."""
import subprocess

import pytest

from polyswift_plusplus_b200 import build_native as B

SOURCE = r"""
#include <cstdio>
#include "sweep_cluster.cuh"
using namespace psb;
template <typename T, int NX, int NY, int NZ, int CL> void row() {
  using P = SweepCl<T, NX, NY, NZ, CL>;
  printf("%d %d %d %d %d %d %d", (int)sizeof(T), NX, NY, NZ, CL, P::NCOL, P::COLS);
  for (int m = 0; m <= CL; ++m) printf(" %d", P::col0(m));
  for (int c = 0; c < P::NCOL; ++c) printf(" %d", P::owner(c));
  printf("\n");
}
int main() {
#define PSB_X(NX, NY, NZ, CL) row<float, NX, NY, NZ, CL>(); row<double, NX, NY, NZ, CL>();
  PSB_SWEEP_GRIDS(PSB_X)
}
"""


@pytest.fixture(scope="module")
def layouts(tmp_path_factory):
    d = tmp_path_factory.mktemp("columns")
    (d / "columns.cu").write_text(SOURCE)
    subprocess.run([B.nvcc_path(), str(d / "columns.cu"), "-o", str(d / "columns"), "-I", str(B.CSRC)]
                   + B._flags(), check=True, capture_output=True, text=True)
    out = subprocess.run([str(d / "columns")], check=True, capture_output=True, text=True).stdout
    return [[int(x) for x in line.split()] for line in out.splitlines()]


def test_every_cta_owns_columns(layouts):
    assert len(layouts) >= 24
    for size, nx, ny, nz, cl, ncol, cols, *rest in layouts:
        first, owner = rest[:cl + 1], rest[cl + 1:]
        assert ncol == ny * (nz // 2 + 1) and first[0] == 0 and first[-1] == ncol and len(owner) == ncol
        for m in range(cl):
            assert 1 <= first[m + 1] - first[m] <= cols, (nx, ny, nz, m)
            assert owner[first[m]:first[m + 1]] == [m] * (first[m + 1] - first[m]), (nx, ny, nz, m)
