"""Operators on layers whose byte offsets pass 2^32: the pattern of a small grid,
repeated along y, gives the small grid's result in every repeat.  GPU only; some 20 GB
on the device."""
import pytest

from native import fine_op

pytestmark = pytest.mark.gpu

PERIOD = 100  # rows of a repeat


def repeats(torch, small, rows):
    """(nz, PERIOD, ...) repeated along y to `rows` rows."""
    n = (rows + PERIOD - 1) // PERIOD
    return small.repeat(1, n, *[1] * (small.ndim - 2))[:, :rows].contiguous()


def test_fp64_layer_beyond_32_bits(tg):
    """14,000 x 13,000 x 1: 182,027,001 nodes a layer, of 24 bytes.  141 operations an
    element at 2^-53, relative to the largest entry."""
    import torch
    nx, ny = 14000, 13000
    gen = torch.Generator("cuda").manual_seed(5)
    ef = torch.rand(1, PERIOD, nx, dtype=torch.float64, device="cuda", generator=gen) + 1e-3
    x = torch.randn(2, PERIOD, nx + 1, 3, dtype=torch.float64, device="cuda", generator=gen)

    def apply(rows):
        y = torch.full((2, rows + 1, nx + 1, 3), torch.nan, dtype=torch.float64, device="cuda")
        fine_op(tg, 0, (nx, rows, 1), repeats(torch, ef, rows), None, repeats(torch, x, rows + 1),
                None, None, 0.0, y)
        return y

    want = apply(3 * PERIOD)[:, PERIOD:2 * PERIOD].clone()
    bound = 1e-13 * want.abs().max()
    got = apply(ny)
    for r in range(PERIOD, ny, PERIOD):
        assert (got[:, r:r + PERIOD] - want).abs().max() < bound, r
    del got
    torch.cuda.empty_cache()


def test_fp32_periodic_layer_beyond_32_bits(tg):
    """A periodic cell of 20,000 x 18,000 x 1: 360,000,000 nodes of 12 bytes.  FP32
    schedules are held to 2e-6."""
    import torch
    from native import I, ModalConsts, call
    nx, ny = 20000, 18000
    gen = torch.Generator("cuda").manual_seed(6)
    ef = torch.rand(1, PERIOD, nx, device="cuda", generator=gen) + 1e-3
    x = torch.randn(1, PERIOD, nx, 3, device="cuda", generator=gen)

    def apply(rows):
        y = torch.full((1, rows, nx, 3), torch.nan, device="cuda")
        call(tg, "_ZN2tg18launch_periodic_opIfEEviiiiRKNS_11ModalConstsEPKT_PKhS6_S6_PS4_Pdii"
             "PKiP11CUstream_st", I(0), I(nx), I(rows), I(1), ModalConsts(), repeats(torch, ef, rows),
             None, repeats(torch, x, rows), None, y, None, I(1), I(1), None, None)
        return y

    want = apply(PERIOD)
    bound = 2e-6 * want.abs().max()
    got = apply(ny)
    for r in range(0, ny, PERIOD):
        assert (got[:, r:r + PERIOD] - want).abs().max() < bound, r
    del got
    torch.cuda.empty_cache()
