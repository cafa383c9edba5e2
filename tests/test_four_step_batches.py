"""Four-step transforms of powers of two where the split's rule changes: a
first factor of 256 up to 2^19 in ComplexF64, balanced splits else.  Against numpy's FP64
transform within 4 eps log2 n, and a column of a batch equal to the transform of
it alone."""
import numpy as np
import pytest

import ffta_b200 as F

pytestmark = pytest.mark.gpu

EPS = {"complex64": 2.0 ** -23, "complex128": 2.0 ** -52}


def check(n, batch, dtype, rows):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n + batch)
    dt = getattr(torch, dtype)
    t = torch.randn((batch, n), dtype=dt, device="cuda", generator=g)
    p = F.plan_fft(t.T, 1)
    y = torch.empty_like(t)
    F.mul_(y.T, p, t.T)
    for r in rows:
        x = t[r].clone()
        ref = np.fft.fft(x.cpu().numpy().astype(np.complex128))
        err = np.linalg.norm(y[r].cpu().numpy() - ref) / np.linalg.norm(ref)
        assert err <= 4 * EPS[dtype] * np.log2(n), (n, batch, r, err)
        assert torch.equal(F.plan_fft(x) * x, y[r]), (n, batch, r)
    return p.describe(t.T)


@pytest.mark.parametrize("dtype", ["complex64", "complex128"])
@pytest.mark.parametrize("batch", [1, 3, 16])
@pytest.mark.parametrize("k", [16, 17, 18, 19, 20])
def test_powers_of_two(k, batch, dtype):
    d = check(1 << k, batch, dtype, sorted({0, batch - 1}))
    assert ("N1=256 " in d) == (k <= (19 if dtype == "complex128" else 17)), d
