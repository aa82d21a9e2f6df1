"""Mixed solves on grids whose level 1 has more than 32,768 nodes, where the V-cycle
applies it without its matrix, against the same solve with the assembled stencil (the
counts of inner iterations stay close) and against the FP64 solution.  GPU only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(128, 64, 64), (127, 63, 65)])
def test_solve_with_and_without_the_matrix(tg, dims):
    from test_gpu_parity import smooth_modulus
    pb = tg.Problem.cantilever(*dims)
    E = smooth_modulus(pb)

    def solve(**options):
        n = tg.kernel_launches()
        u, info = tg.fea_solve_mgcg_matfree(pb, E, tolerance=1e-10, max_iterations=600,
                                            options=tg.SolveOptions(coarsening=2, **options))
        assert info.converged and not info.mixed_fallback, info
        return u, info.iterations, tg.kernel_launches() - n

    u64, _, _ = solve()
    runs = {}
    try:
        for on in (True, False):
            tg.set_level1_tc(on)
            runs[on] = solve(precision=tg.PREC_MIXED)
            assert np.abs(runs[on][0] - u64).max() < 1e-8 * np.abs(u64).max()
    finally:
        tg.set_level1_tc(True)
    its = {on: run[1] for on, run in runs.items()}
    assert abs(its[True] - its[False]) <= max(2, its[False] // 10), its
    # Two launches an application without the matrix, one with it: the switch did act.
    per = {on: run[2] / run[1] for on, run in runs.items()}
    assert per[True] > per[False] + 1.0, per
