"""The step plane pass (variant bit 0) and the x pass in registers (bit 1) over every plane
shape and x extent they exist for, and the one-launch sweeps (both bits) over every grid that
has them, against the passes they replace (variant 0: the shared-memory plane pass, or row
and y-pencil passes where no such pass exists) and, on an uneven grid, against the FP64 oracle.

Tolerances: both paths compute the same transforms with another order of operations.  FP64:
about 2 Ns log2(N) roundings of 1e-16, below 1e-12 of the field's maximum.  FP32 sweeps: a
transform pair's error is about 1e-7 of the maximum and adds up over the 40 steps of two
sweeps as a random walk, below 5e-6.
"""
import math

import numpy as np
import pytest

import oracle as O
from polyswift_plusplus_b200 import workloads as W
from polyswift_plusplus_b200.scft import ScftSolver

pytestmark = pytest.mark.gpu
EXTENTS = (16, 24, 32, 48, 64, 96, 128)


def _case(n, precision, ns=20):
    """A diblock with joints inside the sweep (wfac_in != wfac_out), odd and even step counts."""
    cfg = W.diblock_config(16, 2.0, 0.35, 20.0, ns, W.Updater(kind="steepestDescent", relaxlambdas=(0.1, 0.05)),
                           precision)
    cfg.n = tuple(n)
    cfg.cell = (0.11, 0.07, 0.05)
    x, y, z = W.coords(cfg)
    c = (np.cos(2 * math.pi * x / cfg.box[0]) + np.cos(4 * math.pi * y / cfg.box[1])
         + np.cos(6 * math.pi * z / cfg.box[2])).reshape(-1)
    w = W.random_fields(cfg, 0.3)
    return cfg, [w[0] + c, w[1] - c]


def _fields(cfg, w, variant):
    s = ScftSolver(cfg)
    s.set_variant(variant)
    s.restore(w)
    s.update(2)  # one eager iteration and one from the graph
    out = [s.w(0), s.w(1), s.phi(0), s.phi(1), s.pressure()]
    q = s.scalars()["q"][0]
    s.close()
    return out, q


def _compare(n, precision, variants, against):
    tol = 1e-12 if precision == "fp64" else 5e-6
    cfg, w = _case(n, precision)
    ref, qr = _fields(cfg, w, against)
    for v in variants:
        got, q = _fields(cfg, w, v)
        assert abs(q - qr) <= tol * qr, (n, v)
        for a, b in zip(got, ref):
            assert np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max()), (n, precision, v)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("ny", EXTENTS)
def test_every_plane_shape(gpu, ny, precision):
    for nz in EXTENTS:
        _compare((4, ny, nz), precision, [3, 11], 0)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_every_x_extent(gpu, precision):
    """x extents with their own butterfly split, whole and partial column tiles (12 x 7 columns
    of the row-pass grid), on the compact layout (variant 3) and the plain one (2)."""
    for nx in (1, 4, 8, 12, 16, 24, 32, 48, 64, 96, 128, 256):
        _compare((nx, 16, 24), precision, [2, 3], 0)
        _compare((nx, 12, 12), precision, [2], 0)


@pytest.mark.parametrize("precision,tol", [("fp64", 1e-10), ("mixed", 1e-5)])
def test_uneven_grid_matches_oracle(gpu, oracle_lib, precision, tol):
    cfg, w = _case((12, 48, 32), precision)
    got, q = _fields(cfg, w, 3)
    o = O.Oracle(cfg)
    o.restore(w)
    h = o.update(2)
    assert abs(q - h[-1]["q"][0]) <= tol * q
    for a, b in zip(got, [o.w(0), o.w(1), o.phi(0), o.phi(1), o.pressure()]):
        assert np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("nx", [1, 4, 12, 16, 24, 48, 96, 128])
def test_split_step_256(gpu, nx, precision):
    """256 x 256 planes: the y transform split over the two passes (variants 3, 11) against the
    row and y-pencil passes, for the x extents' butterfly splits."""
    if nx > 24 and precision == "fp64":
        return  # the same x part as in FP32; kept out for time
    _compare((nx, 256, 256), precision, [3, 11], 0)


ONE_LAUNCH = [(16, 16, 16), (24, 24, 24), (32, 32, 32), (16, 16, 1), (32, 32, 1), (64, 64, 1), (128, 128, 1),
              (8, 8, 8), (12, 12, 12), (24, 24, 1), (48, 48, 1), (96, 96, 1)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("n", ONE_LAUNCH)
def test_one_launch_sweeps(gpu, n, precision):
    """A diblock (a change of block inside each sweep), its shortest blocks, and one launch per
    sweep set or per sweep."""
    for ns in (12, 20, 33):
        tol = 1e-12 if precision == "fp64" else 5e-6
        cfg, w = _case(n, precision, ns)
        cfg.polymers[0].blocks[0].force_block_steps = cfg.polymers[0].blocks[1].force_block_steps = True
        ref, qr = _fields(cfg, w, 0)
        for v in (3, 11):
            got, q = _fields(cfg, w, v)
            assert abs(q - qr) <= tol * qr
            for a, b in zip(got, ref):
                assert np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max()), (n, precision, ns, v)
    s = ScftSolver(cfg)
    s.set_variant(3)
    s.restore(w)
    s.update(2)
    assert s.launches_per_iteration < 20
    s.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_one_launch_sweeps_with_junctions_and_in_a_batch(gpu, precision):
    """Sweeps that start from a junction product, and a batch whose members' sweeps share the
    launches: bit for bit the single runs."""
    from polyswift_plusplus_b200.scft import ScftBatch
    items = [W.star_abc(16, precision=precision), W.star_abc(16, precision=precision, fracs=(0.2, 0.4, 0.4), seed=9)]
    cfg = W.blend(16, 18.0, 0.35, 0.15, precision=precision, seed=12, anderson=False, ns=20)
    items.append((cfg, W.random_fields(cfg, 0.3)))
    tol = 1e-12 if precision == "fp64" else 5e-6
    single = []
    for cfg, w in items:
        out = {}
        for v in (0, 3, 11):
            s = ScftSolver(cfg)
            s.set_variant(v)
            s.restore(w)
            s.update(3)
            out[v] = [s.w(i) for i in range(len(cfg.fields))] + [s.phi(i) for i in range(len(cfg.fields))]
            s.close()
        for v in (3, 11):
            for a, b in zip(out[v], out[0]):
                assert np.abs(a - b).max() <= tol * max(1.0, np.abs(b).max())
        single.append(out)
    for v in (3, 11):
        with ScftBatch([c for c, _ in items]) as b:
            b.set_variant(v)
            for i, (_, w) in enumerate(items):
                b.instance(i).restore(w)
            b.update(3)
            for i, (cfg, _) in enumerate(items):
                nf = len(cfg.fields)
                got = [b.instance(i).w(k) for k in range(nf)] + [b.instance(i).phi(k) for k in range(nf)]
                for a, r in zip(got, single[i][v]):
                    assert np.array_equal(a, r)


def test_one_launch_sweep_wait_timeout_is_reported(gpu, oracle_lib):
    """With a poll limit of 0 every wait of the cluster exchange gives up: the error flag is
    reported, the launch ends and the context stays usable."""
    from polyswift_plusplus_b200 import _abi as A
    cfg, w = _case((16, 16, 16), "fp64")
    s = ScftSolver(cfg)
    s.set_variant(3)
    s.restore(w)
    assert gpu.ps_gpu_set_bulk_wait_limit(0) == A.PS_OK
    try:
        with pytest.raises(A.PsError) as ei:
            s.update(1)
    finally:
        assert gpu.ps_gpu_set_bulk_wait_limit(0xFFFFFFFF) == A.PS_OK
    assert ei.value.code == A.PS_GPU_ERR and "wait limit" in str(ei.value)
    s.close()
    test_one_launch_sweeps(gpu, (16, 16, 16), "fp64")


@pytest.mark.parametrize("n,precision", [((64, 24, 24), "fp64"), ((48, 48, 48), "fp64"), ((96, 32, 64), "mixed")])
def test_tuned_run_matches_forced_variant(gpu, n, precision):
    """The tuned choice (variants timed as graphs, the plane pass perhaps started early) gives what
    the same variant gives when forced, bit for bit: starting early changes no arithmetic."""
    cfg, w = _case(n, precision)
    tuned = ScftSolver(cfg)
    tuned.restore(w)
    tuned.update(4)
    v, _ = tuned.variant()
    forced = ScftSolver(cfg)
    forced.restore(w)
    forced.update(1)  # the iteration before tuning
    forced.set_variant(v)
    forced.update(3)
    for i in range(len(cfg.fields)):
        assert np.array_equal(tuned.w(i), forced.w(i)) and np.array_equal(tuned.phi(i), forced.phi(i))
    assert tuned.scalars()["free_energy"] == forced.scalars()["free_energy"]
    tuned.close()
    forced.close()


@pytest.mark.parametrize("n", [(16, 128, 128), (24, 96, 96), (12, 96, 128)])
def test_tuned_run_with_early_plane_pass(gpu, n):
    """The same for the planes whose pass has an early form."""
    test_tuned_run_matches_forced_variant(gpu, n, "mixed")
