"""The volume passes of the OC updates at the edges of their split (one voxel, one
CTA's 512 voxels and one more, both candidate counts), with the multiplier far
below, near and far above the interval (0, 1) that the bisection starts from.

OC updates are the oracle's bit for bit: every branch is decided under a certified
bound.  Projected ones take the device's tanh; a bisection that ends at 1e-6 of its
multiplier moves a candidate by at most half of that.
"""
import numpy as np
import pytest

from oracle.oracle import cantilever

pytestmark = pytest.mark.gpu

SCALES = [1e-9, 0.3, 1e7]


def fields(dims, scale):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx * ny + nz)
    solid = (rng.random(nx * ny * nz) > 0.1).astype(np.uint8)
    solid[0] = 1
    x = np.where(solid > 0, 0.05 + 0.9 * rng.random(solid.size), 0.0)
    dc = -np.where(solid > 0, rng.random(solid.size) * scale, 0.0)
    return cantilever(nx, ny, nz, solid=solid), solid, x, dc


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("dims", [(1, 1, 1), (8, 8, 8), (19, 9, 3), (33, 16, 16), (64, 128, 129)])
def test_oc_update_is_the_oracles(tg, port, dims, scale):
    if dims[0] == 64 and scale != SCALES[0]:
        pytest.skip("the large grid once")
    o, solid, x, dc = fields(dims, scale)
    pb = tg.Problem(*dims, 1.0, solid)
    got = tg.oc_update(pb, tg.make_density_filter(pb, 1.5), x, dc, 0.3)
    assert np.array_equal(got, port.oc_update(o, x, dc, 0.3))


@pytest.mark.parametrize("scale", SCALES)
@pytest.mark.parametrize("dims", [(1, 1, 1), (16, 16, 1), (19, 9, 3), (33, 16, 16)])
def test_projected_update_is_the_oracles(tg, port, dims, scale):
    o, solid, x, dc = fields(dims, scale)
    pb = tg.Problem(*dims, 1.0, solid)
    xt = port.filter(o, x, 1.5)
    got = tg.oc_update_projected(pb, 1.5, x, xt, dc, 4.0, 0.5, 0.3)
    assert np.abs(got - port.oc_update_projected(o, x, xt, dc, 4.0, 0.3)).max() <= 1e-6
