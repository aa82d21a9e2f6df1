"""The matrix-free level-1 operator at the sizes where its tiles end -- coarse
rows of one warp's columns and one more, one coarse element thick, odd fine axes
under both coarsenings, special elements on both ends -- against the assembled
FP32 stencil, within the 2e-6 FP32 schedules are held to.  GPU only."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(6, 6, 6), (56, 6, 8), (58, 8, 6), (60, 10, 7), (62, 7, 9),
                                  (64, 8, 24), (127, 8, 6), (6, 66, 7), (7, 6, 68)])
@pytest.mark.parametrize("coarsening", [1, 2])  # COARSEN_REFERENCE, COARSEN_ALIGNED
def test_level1_matches_stencil_at_tile_edges(tg, dims, coarsening):
    from topopt_gb300.workloads import cantilever_seeded_load
    bcs, loads = cantilever_seeded_load(*dims, seed=1)
    pb = tg.Problem(*dims, 1.0, None, bcs, loads)
    job = tg.SimpJob(pb, tg.SimpParams(), tg.SimpOptions(
        volume_fraction=0.4, change_tol=0.0, cg_tolerance=1e-6, solve=tg.SolveOptions(
            precision=tg.PREC_MIXED, coarsening=coarsening)))
    job.write_design(np.random.default_rng(5).uniform(0.05, 1.0, pb.nv))
    job.step()
    assert job.check_level1() < 2e-6
    job.close()
