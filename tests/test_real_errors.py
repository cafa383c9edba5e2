"""Errors of real transforms of even length whose half has no one-kernel real
transform, beside those of the complex transform of the same length and type:
the inverse is that transform's real part, bit for bit, and so is its error;
rfft, a transform of half the length and a split rounded about once, has the
same error but for the noise of either (measured 0.95 to 1.05 of it in Float32,
0.79 to 1.09 in Float64 over 95 lengths; a split rounded at every operation had
up to 1.13 and more, a twiddle rounded to Float32 1.2)."""
import numpy as np
import pytest

import ffta_b200 as F

pytestmark = pytest.mark.gpu

CPLX = {np.float32: np.complex64, np.float64: np.complex128}


def err(a, b):
    return float(np.linalg.norm((a - b).ravel()) / np.linalg.norm(b.ravel()))


def mirrored(half, n):
    """The full Hermitian spectrum of half spectra (lines, n/2+1), as
    the transform extends it: stored entries as they are."""
    import torch
    return torch.cat([half, half[:, 1:n - half.shape[1] + 1].flip(1).conj()], 1).resolve_conj()


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [36, 146, 324, 648, 2018, 8198, 27648, 46200, 65536])
def test_inverse_is_the_full_length_one(n, dtype):
    import torch
    batch = max(1, 60000 // n)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((batch, n))
    half = torch.from_numpy(np.fft.rfft(x).astype(CPLX[dtype])).cuda()
    z = (F.plan_irfft(half.T, n, 1) * half.T).T.contiguous()
    full = mirrored(half, n)
    w = (F.plan_ifft(full.T, 1) * full.T).T.contiguous()
    assert torch.equal(z, w.real)
    # against long double: the rounding of the imaginary part is not in it
    ld = np.fft.irfft(half.cpu().numpy().astype(np.clongdouble), n=n)
    assert err(z.cpu().numpy(), ld) <= err(w.cpu().numpy(), ld.astype(np.clongdouble))
    # a strided dimension, bit for bit
    s = half.T.contiguous()  # memory (n/2+1, batch): Julia dims (batch, n/2+1)
    assert torch.equal(F.plan_irfft(s.T, n, 2) * s.T, z)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [36, 146, 324, 648, 2018, 8198, 27648, 46200, 65536])
def test_forward_error(n, dtype):
    import torch
    batch = max(1, 60000 // n)
    x = np.random.default_rng(n + 1).standard_normal((batch, n)).astype(dtype)
    t = torch.from_numpy(x).cuda()
    p = F.plan_rfft(t.T, 1)
    assert "by a complex plan" in p.describe((n, batch))
    ld = np.fft.rfft(x.astype(np.longdouble))
    c = t.to(torch.complex64 if dtype == np.float32 else torch.complex128)
    full = (F.plan_fft(c.T, 1) * c.T).T[:, : n // 2 + 1].cpu().numpy()
    assert err((p * t.T).T.cpu().numpy(), ld) <= 1.12 * err(full, ld)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_infinities_and_nans(dtype):
    """An infinity or a NaN reaches every output of its own line and no other; a sum
    that overflows is an infinity, not a NaN."""
    import torch
    n = 324
    x = np.zeros((6, n), dtype=dtype)
    x[0, 0] = x[1, 1] = np.inf
    x[2, 5] = np.nan
    x[3, :2] = np.finfo(dtype).max
    x[4, 7] = -np.inf
    x[5] = np.random.default_rng(1).standard_normal(n)
    t = torch.from_numpy(x).cuda()
    p = F.plan_rfft(t.T, 1)
    y = (p * t.T).T.cpu().numpy()
    for i in (0, 1, 2, 4):
        assert not np.isfinite(y[i]).any(), i
    assert np.isposinf(y[3, 0].real) and y[3, -1] == 0
    assert np.isposinf(y[3, 1].real) and not np.isnan(y[3, 1].imag)
    one = t[5].clone()
    assert np.array_equal(y[5], (F.plan_rfft(one) * one).cpu().numpy())


# a first, a middle and a last strided dimension of three: the extension reads and
# the real part writes the strides
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [14, 324, 2018])
@pytest.mark.parametrize("dim", [2, 3])
def test_inverse_of_a_strided_dimension_of_three(dim, n, dtype):
    import torch
    shape = [3, 4, 5]  # Julia dims
    shape[dim - 1] = n // 2 + 1
    rng = np.random.default_rng(n + dim)
    h = rng.standard_normal((2, *shape))
    x = torch.from_numpy((h[0] + 1j * h[1]).astype(CPLX[dtype])).cuda()
    x = x.permute(2, 1, 0).contiguous().permute(2, 1, 0)  # column-major memory
    z = F.plan_irfft(x, n, dim) * x
    lines = x.movedim(dim - 1, 0).reshape(n // 2 + 1, -1).T.contiguous()  # one row a line
    want = (F.plan_irfft(lines.T, n, 1) * lines.T).T
    assert torch.equal(z.movedim(dim - 1, 0).reshape(n, -1).T, want)
    ld = np.fft.irfft(lines.cpu().numpy().astype(np.clongdouble), n=n)
    assert err(want.cpu().numpy(), ld) <= 4 * np.finfo(dtype).eps * np.log2(n)
