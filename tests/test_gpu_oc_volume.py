"""The volume pass of the OC bisection adds its threads' double-float terms up to FP64's
accuracy: terms whose sums need all of FP64's 53 bits, five more than a double-float has, come out
exactly, on one warp's voxels and on one CTA's, for both candidate counts.  GPU only."""
import ctypes as C

import numpy as np
import pytest

from native import D, I, L, call

pytestmark = pytest.mark.gpu


class OcCands(C.Structure):  # tg_internal.h
    _fields_ = [("k", I), ("c", D * 16)]


@pytest.mark.parametrize("n,bits", [(1, 23), (2, 23), (17, 23), (32, 23), (33, 20), (250, 20),
                                    (256, 20)])
@pytest.mark.parametrize("k", [1, 8, 9, 16])
def test_sums_of_53_bits(tg, n, bits, k):
    import torch
    unit = 2.0 ** -(24 + bits)  # a term: 1 + low units
    low = np.random.default_rng(n).integers(0, 1 << bits, n) | 1
    pair = np.zeros((n, 2), np.float32)
    pair[:, 0], pair[:, 1] = 1.0, low * unit
    term = torch.from_numpy(pair).cuda()  # both bounds of the clamp
    zero, one = torch.zeros_like(term), torch.zeros_like(term)
    one[:, 0] = 1.0
    part = torch.empty(608 * 16, dtype=torch.float64, device="cuda")
    out = torch.full((16,), torch.nan, dtype=torch.float64, device="cuda")
    count = torch.zeros(16, dtype=torch.int32, device="cuda")
    call(tg, "_ZN2tg22launch_oc_volume_multiEPKdS1_S1_S1_lRKNS_7OcCandsEPdS5_PjP11CUstream_st",
         zero, term, term, one, L(n), OcCands(k, (D * 16)(*[1.0] * 16)), part, out, count, None)
    want = n + int(low.sum()) * unit
    assert int(want / unit) == n * 2 ** (24 + bits) + int(low.sum())  # FP64 holds it
    assert out[:k].tolist() == [want] * k and not count.any()
