"""Calls of the library's internal C++ functions, for kernels that no entry point
reaches by themselves.  Buffers are torch tensors on the GPU; the stream is the
default one."""
import ctypes as C

P, I, L, D, F = C.c_void_p, C.c_int, C.c_int64, C.c_double, C.c_float


class Grid(C.Structure):  # tg_internal.h
    _fields_ = [("nx", I), ("ny", I), ("nz", I), ("h", D), ("nnx", I), ("nny", I), ("nnz", I),
                ("nv", L), ("nnodes", L), ("ndof", L)]

    def __init__(self, nx, ny, nz):
        n = (nx + 1) * (ny + 1) * (nz + 1)
        super().__init__(nx, ny, nz, 1.0, nx + 1, ny + 1, nz + 1, nx * ny * nz, n, 3 * n)


class ModalConsts(C.Structure):
    """Unit spacing (tg_internal.h)."""
    _fields_ = [("L", D * 3), ("M", D * 3), ("kdiag", D)]

    def __init__(self, nu=0.3):
        lam, mu = nu / ((1 + nu) * (1 - 2 * nu)), 0.5 / (1 + nu)
        s = [1 / 16, 1 / 48, 1 / 144]
        super().__init__((D * 3)(*[lam * v for v in s]), (D * 3)(*[mu * v for v in s]), 0.0)


class LoopCond(C.Structure):
    _fields_ = [("h", C.c_ulonglong), ("pap", P), ("thr", P), ("st", P)]


class SumOut(C.Structure):
    _fields_ = [("part", P), ("out", P), ("count", P), ("copy_from", P), ("copy_to", P),
                ("cond", LoopCond)]


class MgDims(C.Structure):
    """A level's extents (tg_multigrid.h)."""
    _fields_ = [(n, I) for n in ("ex", "ey", "ez", "nnx", "nny", "nnz", "align")]

    def __init__(self, ex, ey, ez, align=0):
        super().__init__(ex, ey, ez, ex + 1, ey + 1, ez + 1, align)


def ptr(t):
    return None if t is None else P(t.data_ptr())


def call(tg, symbol, *args):
    """Structures go by reference, tensors and None as pointers."""
    import torch
    f = getattr(tg.lib(), symbol)
    f.restype = None
    torch.cuda.synchronize()
    f(*[C.byref(a) if isinstance(a, C.Structure) else
        ptr(a) if a is None or isinstance(a, torch.Tensor) else a for a in args])
    torch.cuda.synchronize()


def fine_op(tg, mode, dims, ef, kn, x, b, invdiag, omega, y, dot=None):
    """launch_fine_op in the vectors' precision; the mode as tg_internal.h numbers it."""
    import torch
    double = x.dtype == torch.float64
    t = "d" if double else "f"
    call(tg, f"_ZN2tg14launch_fine_opI{t}EEviRKNS_4GridERKNS_11ModalConstsEPKT_PKhS9_S9_S9_S7_PS7_"
         "RKNS_6SumOutEP11CUstream_st", I(mode), Grid(*dims), ModalConsts(), ef, kn, x, b, invdiag,
         (D if double else F)(omega), y, dot or SumOut(), None)
