"""One-butterfly lengths (2, 3, 4, 8, 9, 16), whose packed lines go through
shared memory: batches around a block's 128 lines, in place, and the same bits
from lines that are not packed (which take the threads' own loads)."""
import numpy as np
import pytest

import ffta_b200 as F

pytestmark = pytest.mark.gpu

EPS = {np.complex64: 2.0 ** -23, np.complex128: 2.0 ** -52}


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n", [2, 3, 4, 8, 9, 16])
@pytest.mark.parametrize("batch", [1, 2, 127, 128, 129, 1000])
def test_one_butterfly_lines(n, batch, dtype):
    import torch
    rng = np.random.default_rng(n * 2048 + batch)
    x = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(dtype)
    t = torch.from_numpy(x).cuda()
    for plan, ref in ((F.plan_fft, np.fft.fft(x.astype(np.complex128))),
                      (F.plan_ifft, np.fft.ifft(x.astype(np.complex128)))):
        y = (plan(t.T, 1) * t.T).T
        err = np.linalg.norm(y.cpu().numpy() - ref) / np.linalg.norm(ref)
        assert err <= 4 * EPS[dtype] * max(1.0, np.log2(n)), (n, batch, err)
        z = t.clone()
        F.mul_(z.T, plan(z.T, 1), z.T)
        assert torch.equal(z, y)
        wide = torch.zeros((batch, n + 3), dtype=t.dtype, device="cuda")
        wide[:, :n] = t
        out = torch.zeros_like(wide)
        v, o = wide[:, :n], out[:, :n]
        F.mul_(o.T, plan(v.T, 1), v.T)
        assert torch.equal(o, y) and not out[:, n:].any()
