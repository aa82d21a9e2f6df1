"""The marching operator kernel at the sizes where its tiles end: rows of one
warp's columns and one more, strips and chunks of one node, periodic cells whose
rows share a warp (nx <= 32) or not, in FP64, double-float and FP32, against the
oracle.  GPU only."""
import numpy as np
import pytest

from oracle.oracle import cantilever

pytestmark = pytest.mark.gpu

APPLY_DF = 2  # TG_APPLY_DF
# FP64: 141 operations per element at 2^-53; double-float: the same at 2^-47;
# FP32 as every schedule is held to.  Relative to the largest entry.
BOUNDS = ((0, 1e-13), (APPLY_DF, 1e-12), (1, 2e-6))


@pytest.mark.parametrize("dims", [(1, 1, 1), (29, 2, 3), (30, 6, 2), (31, 7, 5), (32, 8, 4),
                                  (63, 4, 17), (95, 2, 2), (5, 40, 33)])
def test_apply_at_tile_edges(tg, port, dims):
    rng = np.random.default_rng(sum(dims))
    nv = dims[0] * dims[1] * dims[2]
    solid = (rng.random(nv) > 0.15).astype(np.uint8)
    solid[0] = 1
    o = cantilever(*dims, solid=solid)
    pb = tg.Problem(*dims, 1.0, solid)
    u = rng.standard_normal(o.ndof)
    f = rng.random(o.nv) + 1e-3
    ref = port.apply(o, u, f)
    for precision, bound in BOUNDS:
        y = tg.fea_matfree_apply(pb, u, youngs_per_voxel=f, precision=precision)
        assert np.abs(y - ref).max() < bound * np.abs(ref).max(), precision


def test_values_at_untouched_nodes_do_not_spread(tg):
    """Nodes of absent elements only may hold anything: the rest of K u is as if
    they held 0, and they get 0."""
    dims = (37, 9, 6)
    tags = np.ones(dims[::-1], np.uint8)
    tags[2:5, 3:7, 10:20] = 0
    pb = tg.Problem(*dims, 1.0, tags.ravel())
    node = np.zeros((7, 10, 38), bool)
    node[3:5, 4:7, 11:20] = True  # every adjacent element is absent
    rng = np.random.default_rng(3)
    u = rng.standard_normal((7, 10, 38, 3))
    u[node] = 0.0
    for precision, _ in BOUNDS:
        want = tg.fea_matfree_apply(pb, u.ravel(), precision=precision)
        for bad in (np.nan, np.inf, 1e300):
            v = u.copy()
            v[node] = bad
            got = tg.fea_matfree_apply(pb, v.ravel(), precision=precision)
            assert np.array_equal(got, want), (precision, bad)
        assert not want.reshape(u.shape)[node].any()


@pytest.mark.parametrize("dims", [(2, 3, 4), (7, 1, 5), (8, 9, 6), (12, 12, 3), (27, 5, 4),
                                  (32, 6, 5), (33, 4, 3), (45, 7, 2)])
@pytest.mark.parametrize("precision", [0, 1])
def test_periodic_rows_and_wraps(tg, port, dims, precision):
    """Homogenized tensors of cells whose rows share a warp, fill it or span
    several, within the 1e-7 the oracle's tolerance of 1e-10 leaves."""
    rng = np.random.default_rng(sum(dims))
    nx, ny, nz = dims
    cell = (rng.random((nz, ny, nx)) > 0.2).astype(np.uint8)
    cell[0, 0, 0] = 1
    want, _, conv = port.homogenize(nx, ny, nz, solid=cell.ravel(), tol=1e-10)
    assert conv
    got, info = tg.homogenize(cell, tolerance=1e-10, precision=precision)
    assert info["converged"]
    assert np.abs(got[0] - want).max() < 1e-7 * np.abs(want).max()
