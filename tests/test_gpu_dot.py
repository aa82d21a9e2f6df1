"""FP32 dot products add their terms up in FP64 as far as a thread per term goes: terms
of 24 bits whose sums need up to 41 come out exactly, on both sides of one CTA, of one
CTA per SM and of four terms a thread in as many.  GPU only."""
import numpy as np
import pytest

from native import L, SumOut, call, ptr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 256, 257, 38912, 38913, 100000, 155648])
def test_fp32_dot_is_exact(tg, n):
    import torch
    low = np.random.default_rng(n).integers(0, 1 << 23, n)
    b = torch.from_numpy((1.0 + low * 2.0 ** -23).astype(np.float32)).cuda()
    part = torch.empty(608, dtype=torch.float64, device="cuda")
    out = torch.full((1,), torch.nan, dtype=torch.float64, device="cuda")
    count = torch.zeros(1, dtype=torch.int32, device="cuda")
    call(tg, "_ZN2tg12launch_dot_fEPKfS1_lRKNS_6SumOutEP11CUstream_st", torch.ones_like(b), b,
         L(n), SumOut(ptr(part), ptr(out), ptr(count)), None)
    assert out.item() == n + int(low.sum()) * 2.0 ** -23 and not count.any()
