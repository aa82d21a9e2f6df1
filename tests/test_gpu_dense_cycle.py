"""Solves whose last smoothed level is applied as a dense matrix, at the edges of that
form: 3, 5 and 7 columns a CTA, its largest level (1,050 DOFs on 26x8x8) and the first
beyond it (28x8x8), odd grids with both coarsenings, a void pocket, and coarsest
levels with an inverse of 702 and 1,269 DOFs, against the CPU's Jacobi-PCG.  Both solve to 1e-12 of the right-hand side; the condition numbers
of these grids (about 1e4) leave 1e-8 of the displacement."""
import numpy as np
import pytest

from oracle.oracle import cantilever
from test_oracle_mg import smooth_modulus

pytestmark = pytest.mark.gpu

CASES = [((8, 8, 8), False), ((12, 8, 8), False), ((24, 8, 8), False), ((26, 8, 8), False),
         ((28, 8, 8), False), ((11, 7, 9), False), ((40, 16, 16), True),
         ((100, 8, 8), False), ((60, 30, 8), False)]


@pytest.mark.parametrize("coarsening", [1, 2])
@pytest.mark.parametrize("dims,voids", CASES)
def test_dense_cycle_solve(tg, port, dims, voids, coarsening):
    nx, ny, nz = dims
    solid = None
    if voids:
        s = np.ones((nz, ny, nx), np.uint8)
        s[4:10, 4:10, 10:20] = 0
        solid = s.ravel()
    o = cantilever(nx, ny, nz, solid=solid)
    pb = tg.Problem(nx, ny, nz, 1.0, solid, list(zip(o.bc_node, o.bc_comp, o.bc_val)),
                    list(zip(o.ld_node, o.ld_comp, o.ld_val)))
    f = smooth_modulus(*dims)
    ue, _, _ = port.solve_cg(o, f, tol=1e-12)
    for prec in (0, tg.PREC_MIXED):
        u, info = tg.fea_solve_mgcg_matfree(pb, f, tolerance=1e-12, max_iterations=2000,
                                            options=tg.SolveOptions(precision=prec,
                                                                    coarsening=coarsening))
        assert info.converged and info.mg_levels >= 3
        assert np.abs(u - ue).max() <= 1e-8 * np.abs(ue).max()


def test_dense_cycles_from_many_threads(tg):
    """Hierarchies with dense levels of different sizes built at the same time: each
    solve is the one it is alone, bit for bit."""
    from concurrent.futures import ThreadPoolExecutor
    dims = [(8, 8, 8), (12, 8, 8), (16, 8, 8), (20, 8, 8), (24, 8, 8), (26, 8, 8)]
    jobs = [(tg.Problem.cantilever(*d), smooth_modulus(*d)) for d in dims]

    def solve(i):
        pb, f = jobs[i % len(jobs)]
        return tg.fea_solve_mgcg_matfree(pb, f, tolerance=1e-6)[0]

    alone = [solve(i) for i in range(len(jobs))]
    with ThreadPoolExecutor(6) as pool:
        for i, u in enumerate(pool.map(solve, range(60))):
            assert np.array_equal(u, alone[i % len(jobs)])
