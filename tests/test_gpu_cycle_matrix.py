"""The last smoothed level's V-cycle as a dense matrix, against the same cycle in plain
FP64 on the CPU: a random symmetric stencil, inactive DOFs on both levels, even and odd
axes under both coarsenings, damped Jacobi with one and two sweeps and Chebyshev of degree
3 and 4, and the three counts of columns a CTA.

An entry is a chain of about a thousand operations (81 a row and smoothing step, up to
nine steps, the coarsest solve's row), none of which grows: at 2^-53 in FP64 and 2^-46 in
the double-float arithmetic of FP32 hierarchies, 1e-12 and 1e-10 of the largest entry.
GPU only."""
import numpy as np
import pytest

from native import D, F, I, MgDims, call

pytestmark = pytest.mark.gpu


def stencil(rng, dims, act, real):
    """The 14 stored blocks [126][nodes] and the dense matrix they are half of."""
    nnx, nny, nnz = (e + 1 for e in dims)
    nn = nnx * nny * nnz
    A, K = np.zeros((126, nn), real), np.zeros((3 * nn, 3 * nn))
    for j in range(14):
        di = 13 + j
        dx, dy, dz = di % 3 - 1, di // 3 % 3 - 1, di // 9 - 1
        for n in range(nn):
            a, b, c = n % nnx + dx, n // nnx % nny + dy, n // (nnx * nny) + dz
            if not (0 <= a < nnx and 0 <= b < nny and 0 <= c < nnz):
                continue
            m = (c * nny + b) * nnx + a
            blk = rng.uniform(-1.0, 1.0, (3, 3)).astype(real)
            if j == 0:
                blk = blk + blk.T + real(90.0) * np.eye(3, dtype=real)
            blk = blk * np.outer(act[3 * n:3 * n + 3], act[3 * m:3 * m + 3])
            A[9 * j:9 * j + 9, n] = blk.ravel()
            K[3 * n:3 * n + 3, 3 * m:3 * m + 3] = blk
            K[3 * m:3 * m + 3, 3 * n:3 * n + 3] = blk.T if j else blk
    return A, K


def axis_prolongation(ef, align):
    p = np.zeros((ef + 1, (ef + 1) // 2 + 1))
    for i in range(ef + 1):
        if align and ef % 2 and i == ef:
            p[i, (i + 1) // 2] = 1.0
        elif i % 2 == 0:
            p[i, i // 2] = 1.0
        else:
            p[i, i // 2] = p[i, i // 2 + 1] = 0.5
    return p


def cycle(K, act, dinv, P, Ainv, coef, degree, sweeps, omega):
    b = np.eye(len(K))
    dinv, act = dinv[:, None], act[:, None]
    x, step, direction = np.zeros_like(K), degree or sweeps, None
    for half in range(2):
        for k in range(step):
            res = dinv * (b - K @ x)
            if degree:
                direction = coef[0] * res if k == 0 else coef[2 * k] * direction + coef[2 * k + 1] * res
                x = x + act * direction
            else:
                x = x + act * omega * res
        if half == 0:
            x = x + act * (P @ (Ainv @ (P.T @ (act * (b - K @ x)))))
    return x


@pytest.mark.parametrize("real,bound", [(np.float64, 1e-12), (np.float32, 1e-10)])
@pytest.mark.parametrize("degree,sweeps", [(0, 1), (0, 2), (3, 1), (4, 1)])
@pytest.mark.parametrize("dims,align", [((3, 3, 3), 0), ((4, 4, 4), 0), ((5, 3, 4), 1),
                                        ((7, 5, 3), 0), ((8, 4, 4), 0), ((13, 4, 4), 1)])
def test_cycle_matrix(tg, dims, align, degree, sweeps, real, bound):
    import torch
    rng = np.random.default_rng(sum(dims) + degree)
    coarse = [(e + 1) // 2 for e in dims]
    nn, cnn = np.prod([e + 1 for e in dims]), np.prod([e + 1 for e in coarse])
    act = (rng.random(3 * nn) > 0.1).astype(np.uint8)
    cact = rng.random(3 * cnn) > 0.2
    A, K = stencil(rng, dims, act, real)
    dinv = np.where(act > 0, 1.0 / np.where(act > 0, np.diag(K), 1.0), 0.0).astype(real)
    px, py, pz = (axis_prolongation(e, align) for e in dims)
    P = np.kron(np.kron(np.kron(pz, py), px), np.eye(3))[:, cact]
    nc = P.shape[1]
    g = rng.standard_normal((nc, nc))
    Ainv = (g + g.T) / (40.0 * np.sqrt(nc))
    coef = rng.uniform(0.1, 0.9, 16).astype(np.float32)
    omega = real(0.6)
    want = cycle(K, act, dinv.astype(np.float64), P, Ainv, coef.astype(np.float64), degree, sweeps,
                 float(omega))
    cidx = np.full(3 * cnn, -1, np.int32)
    cidx[cact] = np.arange(nc)
    dev = [torch.from_numpy(np.ascontiguousarray(v)).cuda()
           for v in (A, act, dinv, coef, Ainv, cidx, np.flatnonzero(cact).astype(np.int32))]
    M = torch.full((3 * nn, 3 * nn), torch.nan, dtype=torch.float64, device="cuda")
    t, scalar = ("d", D) if real is np.float64 else ("f", F)
    call(tg, f"_ZN2tg14mg_dense_cycleI{t}EEvRKNS_6MgDimsES3_PKT_PKhS6_PKfiiS4_PKdiPKiSE_Pd"
         "P11CUstream_st", MgDims(*dims, align), MgDims(*coarse, align), dev[0], dev[1], dev[2],
         dev[3], I(degree), I(sweeps), scalar(omega), dev[4], I(nc), dev[5], dev[6], M, None)
    assert np.abs(M.cpu().numpy() - want).max() <= bound * np.abs(want).max()
