"""The fine operator as the solvers run it -- product, residual and smoothing sweep on
the kept DOFs, with the sums that ride in the product and the sweep -- in FP64 on both
sides of its choice of kernel and in FP32, at rows of one warp's columns and one more,
against the oracle's product.  192 operations an element at 2^-53, and the 2e-6 that FP32
schedules are held to, relative to the largest entry (of the sums: to their terms'
magnitudes).  GPU only."""
import numpy as np
import pytest

from native import SumOut, fine_op, ptr
from oracle.oracle import cantilever

pytestmark = pytest.mark.gpu

APPLY, RESIDUAL, SMOOTH = 0, 1, 2
OMEGA = 0.6


@pytest.mark.parametrize("double", [True, False])
@pytest.mark.parametrize("dims", [(1, 1, 1), (24, 8, 8), (48, 8, 8), (30, 4, 3), (31, 5, 4),
                                  (62, 9, 7), (3, 3, 40), (60, 20, 20)])
def test_modes_on_kept_dofs(tg, port, dims, double):
    import torch
    real, bound = (np.float64, 1e-13) if double else (np.float32, 2e-6)
    rng = np.random.default_rng(dims[0] + dims[2])
    nx, ny, nz = dims
    solid = (rng.random((nz, ny, nx)) > 0.1).astype(np.uint8)
    solid[0, 0, 0] = 1
    o = cantilever(*dims, solid=solid.ravel())
    f = ((rng.random(solid.shape) + 1e-3) * solid).astype(real)
    touched = np.zeros((nz + 1, ny + 1, nx + 1), bool)
    for c in range(8):
        z, y, x = c >> 2, (c >> 1) & 1, c & 1
        touched[z:z + nz, y:y + ny, x:x + nx] |= solid > 0
    kept = touched[..., None] & (rng.random(touched.shape + (3,)) > 0.1)
    node = (kept * np.array([1, 2, 4])).sum(-1).astype(np.uint8)
    keep = kept.ravel()
    u, b, d = (rng.standard_normal(o.ndof).astype(real) for _ in range(3))
    u, d = u * keep, np.abs(d) * keep
    u64, b64, d64 = (v.astype(np.float64) for v in (u, b, d))
    au = port.apply(o, u64, f.ravel().astype(np.float64))
    want = {APPLY: au * keep, RESIDUAL: (b64 - au) * keep,
            SMOOTH: (u64 + OMEGA * d64 * (b64 - au)) * keep}
    dev = {k: torch.from_numpy(np.ascontiguousarray(v)).cuda()
           for k, v in dict(f=f, node=node, u=u, b=b, d=d).items()}
    part = torch.empty(1 << 18, dtype=torch.float64, device="cuda")
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    for mode, ref in want.items():
        y = torch.full_like(dev["u"], torch.nan)
        out = torch.full((1,), torch.nan, dtype=torch.float64, device="cuda")
        dot = None if mode == RESIDUAL else SumOut(ptr(part), ptr(out), ptr(count))
        fine_op(tg, mode, dims, dev["f"], dev["node"], dev["u"], dev["b"], dev["d"], OMEGA, y, dot)
        got = y.cpu().numpy()
        assert np.abs(got - ref).max() <= bound * np.abs(ref).max(), mode
        assert not got[~keep].any(), mode
        if dot is not None:
            terms = (u64 if mode == APPLY else b64) * ref
            assert abs(out.item() - terms.sum()) <= bound * np.abs(terms).sum(), mode
            assert not count.any()
