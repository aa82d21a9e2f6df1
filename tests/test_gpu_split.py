"""The FP64 operator on both sides of its choice of kernel -- a warp per element row and
component on small grids, the marching kernel where rows fill the SMs -- at rows of one
warp's columns and one more, strips and chunks that end with the grid, against the
oracle: 192 operations an element at 2^-53, relative to the largest entry."""
import numpy as np
import pytest

from oracle.oracle import cantilever

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(24, 8, 8), (48, 8, 8), (30, 4, 3), (31, 5, 4), (62, 9, 7),
                                  (3, 3, 40), (60, 20, 20), (60, 36, 28), (96, 48, 48)])
def test_fp64_operator(tg, port, dims):
    rng = np.random.default_rng(dims[0])
    nv = dims[0] * dims[1] * dims[2]
    solid = (rng.random(nv) > 0.1).astype(np.uint8)
    solid[0] = 1
    o = cantilever(*dims, solid=solid)
    pb = tg.Problem(*dims, 1.0, solid)
    u, f = rng.standard_normal(o.ndof), rng.random(o.nv) + 1e-3
    ref = port.apply(o, u, f)
    got = tg.fea_matfree_apply(pb, u, youngs_per_voxel=f)
    assert np.abs(got - ref).max() < 1e-13 * np.abs(ref).max()
