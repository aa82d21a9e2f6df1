"""The Jacobi-PCG on both sides of the size where its preconditioned residual rides in
the update of r (155,648 DOFs: 26x43x43 below, 26x43x44 above), odd and even DOF counts,
against the CPU's (both to 1e-12 of the right-hand side; condition numbers of about 1e4
leave 1e-8 of the displacement), and the loop in a graph against the host's, bit for
bit."""
import numpy as np
import pytest

from oracle.oracle import cantilever
from test_oracle_mg import smooth_modulus

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(2, 2, 2), (9, 6, 4), (24, 8, 8), (26, 43, 43), (26, 43, 44)])
def test_jacobi_pcg(tg, port, dims):
    o = cantilever(*dims)
    pb = tg.Problem.cantilever(*dims)
    f = smooth_modulus(*dims)
    want, _, _ = port.solve_cg(o, f, tol=1e-12)
    got = [tg.fea_solve_mgcg_matfree(pb, f, tolerance=1e-12, options=tg.SolveOptions(
        solver=1, graph_mode=mode)) for mode in (0, tg.GRAPH_OFF)]
    (u, info), (uh, ih) = got
    assert info.converged and not info.used_multigrid
    assert np.abs(u - want).max() <= 1e-8 * np.abs(want).max()
    assert np.array_equal(u, uh) and info.iterations == ih.iterations
