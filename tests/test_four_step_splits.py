"""Splits of lengths that have both a prime of 17..71 and a factor for
Bluestein: the prime joins the Bluestein factor where a prime stage of its own
would cost more.  Against numpy's FP64 transform within 4 eps log2 n."""
import re

import numpy as np
import pytest

import ffta_b200 as F

pytestmark = pytest.mark.gpu


# 29252 = 4 * 71 * 103, 5871 = 3 * 19 * 103, 6142 = 2 * 37 * 83, 196725 =
# 25 * 3 * 43 * 61 (Bluestein though 43 and 61 have stages: two such passes cost
# more); 5301 = 9 * 19 * 31 has no Bluestein split
@pytest.mark.parametrize("n,dtype,n1", [
    (29252, np.complex64, 4), (5871, np.complex64, 3), (6142, np.complex64, 2),
    (196725, np.complex64, 25), (5301, np.complex64, 57), (5871, np.complex128, 3),
    (6142, np.complex128, 2), (5301, np.complex128, 57)])
def test_prime_joins_the_bluestein_factor(n, dtype, n1):
    import torch
    rng = np.random.default_rng(n)
    x = (rng.standard_normal((3, n)) + 1j * rng.standard_normal((3, n))).astype(dtype)
    t = torch.from_numpy(x).cuda()
    p = F.plan_fft(t.T, 1)
    assert f"N1={n1} " in p.describe(t.T), p.describe(t.T)
    y = (p * t.T).T.cpu().numpy()
    ref = np.fft.fft(x.astype(np.complex128))
    assert np.linalg.norm(y - ref) <= 4 * np.finfo(dtype).eps * np.log2(n) * np.linalg.norm(ref)


# first factors of 2, 3 and 4: 64 of their columns to a block where that gives
# 148 blocks (not a multiple of 64, contiguous and strided lines), else fewer
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n,n1,batch", [(1942, 2, 11), (321, 3, 95), (26244, 4, 2), (1942, 2, 1)])
def test_short_first_factor(n, n1, batch, dtype):
    import torch
    rng = np.random.default_rng(n + batch)
    x = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(dtype)
    ref = np.fft.fft(x.astype(np.complex128))
    bound = 4 * np.finfo(dtype).eps * np.log2(n) * np.linalg.norm(ref)
    t = torch.from_numpy(x).cuda()
    p = F.plan_fft(t.T, 1)
    full = batch * n // n1 >= 64 * 148
    assert re.search(rf"\.1\(N1={n1} L={n1} [^)]*\)\[tile T=1 G={64 if full else ""}", p.describe(t.T))
    assert np.linalg.norm((p * t.T).T.cpu().numpy() - ref) <= bound
    s = t.T.contiguous()  # memory (n, batch): Julia dims (batch, n)
    assert np.linalg.norm((F.plan_fft(s.T, 2) * s.T).cpu().numpy() - ref) <= bound
