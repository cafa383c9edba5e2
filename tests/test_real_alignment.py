"""Real arrays that are aligned to one real only (an address in the middle of
a complex value), of lengths whose half has a one-kernel real transform: the
C ABI takes them, and a slice of a tensor gives them.  Same operations on the
same values, so the same bits as for an aligned array."""
import ctypes

import numpy as np
import pytest

import ffta_b200 as F
from ffta_b200 import _lib

pytestmark = pytest.mark.gpu


def _execute(h, src, dst):
    import torch
    rc = _lib.lib.fb_execute(h, ctypes.c_void_p(src.data_ptr()), ctypes.c_void_p(dst.data_ptr()),
                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == _lib.FB_OK, _lib.last_error()


# one butterfly per thread, several lines per block, the split in registers
# and through shared memory, 1024 threads a line; one line and a ragged batch
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("batch", [1, 7])
@pytest.mark.parametrize("n", [4, 18, 32, 64, 250, 1000, 4096, 8192])
def test_lines_at_an_odd_real(n, batch, dtype):
    import torch
    rng = np.random.default_rng(n + batch)
    x = torch.from_numpy(rng.standard_normal((batch, n)).astype(dtype)).cuda()
    buf = torch.full((batch * n + 3,), 7.0, dtype=x.dtype, device="cuda")
    off = buf[1:1 + batch * n].view(batch, n)
    assert x.data_ptr() % (2 * x.element_size()) == 0
    assert off.data_ptr() % (2 * x.element_size()) != 0
    off.copy_(x)
    p = F.plan_rfft(x.T, 1)
    assert "REAL-HALF(L=" in p.describe((n, batch)) and "complex plan" not in p.describe((n, batch))
    y = p * x.T
    for _ in range(2):  # the second call takes the repeated-layout path
        assert torch.equal(p * off.T, y)
    q = F.plan_irfft(y, n, 1)
    z = q * y
    off.fill_(3.0)
    _execute(q._handle((n, batch)), y.T.contiguous(), off)
    assert torch.equal(off, z.T)
    assert float(buf[0]) == 7.0 and float(buf[-1]) == 7.0 and float(buf[-2]) == 7.0


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_images_at_an_odd_real(dtype):
    import torch
    n1, n2 = 64, 21
    rng = np.random.default_rng(9)
    x = torch.from_numpy(rng.standard_normal((n2, n1)).astype(dtype)).cuda()
    buf = torch.zeros(n1 * n2 + 1, dtype=x.dtype, device="cuda")
    off = buf[1:].view(n2, n1)
    off.copy_(x)
    p = F.plan_rfft(x.T, (1, 2))
    y = p * x.T
    assert torch.equal(p * off.T, y)
    q = F.plan_irfft(y, n1, (1, 2))
    z = q * y
    _execute(q._handle((n1, n2)), y.T.contiguous(), off)
    assert torch.equal(off, z.T)
