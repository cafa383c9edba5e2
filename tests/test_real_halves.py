"""Real transforms whose half length has no one-kernel real transform: a
complex plan of length n/2 with the split (rfft) or the merge (brfft) as a
pass.  Halves that run on the generic kernel, in four steps and by Bluestein,
one line and several, a strided dimension, two dimensions, and real data that
is not aligned to a complex value.  Against numpy's FP64 transform within
4 eps log2 n; strided equal to contiguous bit for bit."""
import numpy as np
import pytest

import ffta_b200 as F

pytestmark = pytest.mark.gpu

EPS = {np.float32: 2.0 ** -23, np.float64: 2.0 ** -52}


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("batch", [1, 3, 40])
@pytest.mark.parametrize("n", [14, 26, 324, 2 * 1009, 2 * 4099, 32768, 2 * 23100])
def test_halves(n, batch, dtype):
    import torch
    rng = np.random.default_rng(n + batch)
    x = rng.standard_normal((batch, n)).astype(dtype)
    t = torch.from_numpy(x).cuda()
    p = F.plan_rfft(t.T, 1)
    assert "by a complex plan" in p.describe((n, batch))
    y = p * t.T  # (n/2+1, batch)
    bound = 4 * EPS[dtype] * np.log2(n)
    assert rel(y.T.cpu().numpy(), np.fft.rfft(x.astype(np.float64))) <= bound
    q = F.plan_irfft(y, n, 1)
    for _ in range(2):  # the second call takes the repeated-layout path
        assert rel((q * y).T.cpu().numpy(), x) <= 2 * bound
    # a strided dimension, bit for bit
    s = t.T.contiguous()  # memory (n, batch): Julia dims (batch, n)
    ys = F.plan_rfft(s.T, 2) * s.T
    assert torch.equal(ys, y.T)
    zs = F.plan_irfft(ys, n, 2) * ys
    assert torch.equal(zs, (q * y).T)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_two_dimensions(dtype):
    import torch
    rng = np.random.default_rng(3)
    x = rng.standard_normal((2, 21, 260)).astype(dtype)  # Julia dims (260, 21, 2)
    t = torch.from_numpy(x).cuda().permute(2, 1, 0)
    y = F.plan_rfft(t, (1, 2)) * t
    ref = np.fft.rfft2(x.astype(np.float64))
    bound = 4 * EPS[dtype] * np.log2(260 * 21)
    assert rel(y.permute(2, 1, 0).cpu().numpy(), ref) <= bound
    z = F.plan_irfft(y, 260, (1, 2)) * y
    assert rel(z.permute(2, 1, 0).cpu().numpy(), x) <= 2 * bound


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_real_data_aligned_to_one_real(dtype):
    """The C ABI takes real arrays aligned to a real: both directions from and
    to an address in the middle of a complex value."""
    import ctypes

    import torch
    from ffta_b200 import _lib
    n, b = 324, 5
    rng = np.random.default_rng(4)
    x = rng.standard_normal((b, n)).astype(dtype)
    buf = torch.zeros(b * n + 1, dtype=torch.from_numpy(x).dtype, device="cuda")
    buf[1:] = torch.from_numpy(x).cuda().reshape(-1)
    off = buf[1:].reshape(b, n)
    assert off.data_ptr() % (2 * off.element_size()) != 0
    y = F.plan_rfft(off.T, 1) * off.T
    bound = 4 * EPS[dtype] * np.log2(n)
    assert rel(y.T.cpu().numpy(), np.fft.rfft(x.astype(np.float64))) <= bound
    q = F.plan_brfft(y, n, 1)
    h = q._handle((n, b))
    buf.zero_()
    yc = y.T.contiguous()
    rc = _lib.lib.fb_execute(h, ctypes.c_void_p(yc.data_ptr()), ctypes.c_void_p(off.data_ptr()),
                             ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == _lib.FB_OK, _lib.last_error()
    torch.cuda.synchronize()
    assert rel(off.cpu().numpy() / n, x) <= 2 * bound
    assert float(buf[0]) == 0.0


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("batch", [1, 3, 33])
@pytest.mark.parametrize("n", [64, 128, 256, 1024, 2048, 4096, 16384])
def test_split_in_registers(n, batch, dtype):
    """Halves whose last stage holds butterflies in pairs (j and n/2/radix - j)
    split in registers: every output, and a line alone gives the same bits."""
    import torch
    rng = np.random.default_rng(n * 7 + batch)
    x = rng.standard_normal((batch, n)).astype(dtype)
    t = torch.from_numpy(x).cuda()
    p = F.plan_rfft(t.T, 1)
    assert "REAL-HALF(L=" in p.describe((n, batch)) and "complex plan" not in p.describe((n, batch))
    y = (p * t.T).T
    assert rel(y.cpu().numpy(), np.fft.rfft(x.astype(np.float64))) <= 4 * EPS[dtype] * np.log2(n)
    one = t[batch // 2].clone()
    assert torch.equal(F.plan_rfft(one) * one, y[batch // 2])
