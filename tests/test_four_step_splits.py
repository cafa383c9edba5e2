"""Splits of lengths that have both a prime of 17..71 and a factor for
Bluestein: the prime joins the Bluestein factor where a prime stage of its own
would cost more.  Against numpy's FP64 transform within 4 eps log2 n."""
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
