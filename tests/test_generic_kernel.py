"""The generic line kernel at the sizes where its branches change: prime
stages of 17..71 shared by a line's threads (one prime alone, several in one
length, more output pairs per thread than the usual eight), first and last
stages with direct I/O on contiguous and on strided lines, one-stage programs,
lines that leave a block's last group partly empty.  Against the __float128
oracle within 4 eps log2 n (its FP64 run sums a prime leaf with a recurrence
and is itself 6.5e-15 off at n = 59), and strided equal to contiguous bit for
bit."""
import numpy as np
import pytest

import ffta_b200 as F
import oracle

pytestmark = pytest.mark.gpu

EPS = {np.complex64: 2.0 ** -23, np.complex128: 2.0 ** -52}


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n", [7, 11, 13, 17, 59, 71, 2 * 61, 16 * 17, 17 * 71, 231, 1001, 17 ** 3,
                               71 * 71, 71 * 100, 7168])
@pytest.mark.parametrize("batch", [1, 5, 37])
def test_generic_lengths(n, batch, dtype):
    import torch
    rng = np.random.default_rng(n * 64 + batch)
    x = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(dtype)
    t = torch.from_numpy(x).cuda()
    for direction, plan in ((-1, F.plan_fft), (1, F.plan_bfft)):
        p = plan(t.T, 1)
        y = (p * t.T).T.cpu().numpy()
        rows = sorted({0, batch // 2, batch - 1})
        ref = np.stack([oracle.fft_nd(x[r], None, direction, prec="f128") for r in rows])
        err = np.linalg.norm(y[rows] - ref) / np.linalg.norm(ref)
        assert err <= 4 * EPS[dtype] * np.log2(n), (n, direction, err, p.describe(t.T))
        # the same lines along the second dimension, in place
        s = torch.from_numpy(np.ascontiguousarray(x.T)).cuda()
        q = plan(s.T, 2, _flags=F.FB_FLAG_SAME_SCHEDULE_STRIDED)
        F.mul_(s.T, q, s.T)
        assert np.array_equal(s.cpu().numpy().T, y), (n, direction, q.describe(s.T))
