"""The Jacobi-PCG on both sides of the sizes where its update changes: 38,912 DOFs, up
to which a thread takes one entry, and 155,648, up to which the preconditioned residual
rides in the update of r, against the CPU's (both to 1e-12 of the right-hand side;
condition numbers of about 1e4 leave 1e-8 of the displacement), and the loop in a graph
against the host's, bit for bit.  GPU only."""
import numpy as np
import pytest

from oracle.oracle import cantilever
from test_oracle_mg import smooth_modulus

pytestmark = pytest.mark.gpu

ONE, RIDES = 152 * 256, 152 * 1024


@pytest.mark.parametrize("dims,above", [((26, 20, 21), ()), ((26, 21, 21), (ONE,)),
                                        ((26, 42, 43), (ONE,)), ((26, 43, 43), (ONE, RIDES))])
def test_jacobi_pcg_at_its_edges(tg, port, dims, above):
    o = cantilever(*dims)
    assert tuple(n for n in (ONE, RIDES) if o.ndof > n) == above
    pb = tg.Problem.cantilever(*dims)
    f = smooth_modulus(*dims)
    want, _, _ = port.solve_cg(o, f, tol=1e-12)
    (u, info), (uh, ih) = [tg.fea_solve_mgcg_matfree(pb, f, tolerance=1e-12, options=tg.SolveOptions(
        solver=1, graph_mode=mode)) for mode in (0, tg.GRAPH_OFF)]
    assert info.converged and not info.used_multigrid
    assert np.abs(u - want).max() <= 1e-8 * np.abs(want).max()
    assert np.array_equal(u, uh) and info.iterations == ih.iterations
