"""p.Ap of mixed homogenization: a thread's FP32 run covers sixteen nodes at most, as many
layers as its march takes.  A checkerboard field is an eigenvector of the periodic
operator; with one stiff element layer its terms are c / 2 on two node layers and 2^-26 c
on the others, which a run that starts with the stiff ones loses.  Of sixteen nodes'
terms that is 2^-23 of the sum of the two layers.  GPU only."""
import numpy as np
import pytest

from native import I, ModalConsts, call

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [16, 32, 48, 64, 128])
def test_small_terms_are_summed(tg, n):
    import torch
    ef = np.full((n, n, n), 2.0 ** -26, np.float32)
    ef[0] = 1.0
    z, y, x = np.meshgrid(*3 * [np.arange(n)], indexing="ij")
    u = np.zeros((n, n, n, 3), np.float32)
    u[..., 0] = 1 - 2 * ((x + y + z) & 1)
    ef, u = torch.from_numpy(ef).cuda(), torch.from_numpy(u).cuda()
    out = torch.full_like(u, torch.nan)
    blocks = tg.lib()["_ZN2tg18periodic_op_blocksIfEEiiii"](I(n), I(n), I(n))
    part = torch.full((blocks,), torch.nan, dtype=torch.float64, device="cuda")
    call(tg, "_ZN2tg18launch_periodic_opIfEEviiiiRKNS_11ModalConstsEPKT_PKhS6_S6_PS4_Pdii"
         "PKiP11CUstream_st", I(0), I(n), I(n), I(n), ModalConsts(), ef, None, u, None, out, part,
         I(1), I(1), None, None)
    terms = u.double() * out.double()
    assert float(terms.min()) >= 0.0
    assert abs(float(part.sum() - terms.sum())) <= 2.0 ** -23 * float(terms.sum())
