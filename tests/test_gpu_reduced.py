"""The reduced system of grids with void voxels, repeated loads and boundary
conditions and prescribed displacements, at one element row, odd rows and a grid whose
setup runs on several host threads (104x101x101 nodes): the kept set and its size are
the oracle's, and so is the right-hand side, bit for bit without prescribed values
(loads add up in their order) and within 1e-12 of its largest entry with them (K u_p is
summed in another order)."""
import numpy as np
import pytest

from oracle.oracle import Problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prescribed", [False, True])
@pytest.mark.parametrize("dims", [(1, 1, 1), (9, 1, 2), (7, 5, 6), (103, 100, 100)])
def test_reduced_system(tg, port, dims, prescribed):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    solid = (rng.random(nx * ny * nz) > 0.2).astype(np.uint8)
    solid.reshape(nz, ny, nx)[:, :, [0, -1]] = 1
    node = Problem(nx, ny, nz).node
    bcs = [(node(0, b, c), k, 0.01 * b if prescribed and k == 1 else 0.0)
           for c in range(nz + 1) for b in range(ny + 1) for k in range(3)]
    bcs += bcs[:5]
    loads = [(node(nx, b, nz), 2, 0.1 * (b + 1)) for b in range(ny + 1)]
    loads += [(node(nx, 0, nz), 2, -0.7), (node(nx, ny, 0), 0, 1.5), (node(nx, 0, nz), 2, 1e-3)]
    want = port.build_reduced(Problem(nx, ny, nz, 1.0, solid, bcs, loads))
    got = tg.fea_build_reduced(tg.Problem(nx, ny, nz, 1.0, solid, bcs, loads), None)
    assert got["ng"] == want["ng"]
    assert np.array_equal(got["kept"], want["kept"])
    if prescribed:
        assert np.abs(got["rhs"] - want["rhs"]).max() <= 1e-12 * np.abs(want["rhs"]).max()
    else:
        assert np.array_equal(got["rhs"], want["rhs"])
