"""Strided lines whose elements are more than 2^31 array elements apart from first
to last: they keep the tile kernels, whose steps between the elements of a
butterfly are 32-bit and whose other offsets 64-bit, while those steps fit.  Same bits as
contiguous lines of the same values."""
import numpy as np
import pytest

import ffta_b200 as F

pytestmark = pytest.mark.gpu


def need(gigabytes):
    import torch
    free, _ = torch.cuda.mem_get_info()
    if free < gigabytes * 1e9:
        pytest.skip(f"needs {gigabytes} GB of device memory")


def columns(count, n, dtype, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    real = torch.float32 if dtype == torch.complex64 else torch.float64
    return torch.view_as_complex(torch.randn((count, n, 2), generator=g, device="cuda", dtype=real))


# (n, elements from one element of a line to the next): line ends 2^31 and more
# apart; in the last case (last radix 3) steps too, which the generic kernel runs
@pytest.mark.parametrize("n,stride,gb", [(1024, (1 << 21) + 24, 18), (4096, (1 << 20) + 8, 35),
                                         (27, 100000007, 22), (48, (1 << 27) + 8, 52)])
@pytest.mark.parametrize("generic", [False, True])
def test_strided_lines(n, stride, gb, generic):
    import torch
    need(gb + 4)
    torch.cuda.empty_cache()
    count = 9
    cols = columns(count, n, torch.complex64, n)
    ref = (F.plan_fft(cols.T, 1) * cols.T).T
    big = torch.empty(((n - 1) * stride + count,), dtype=torch.complex64, device="cuda")
    view = big.as_strided((count, n), (1, stride))  # Julia dims (count, n)
    view.copy_(cols)
    p = F.plan_fft(view, 2,
                   _flags=F.FB_FLAG_SAME_SCHEDULE_STRIDED | (F.FB_FLAG_GENERIC_ONLY if generic else 0))
    if not generic:
        assert ("[tile" in p.describe(view)) == (n != 48), p.describe(view)
    F.mul_(view, p, view)
    assert torch.equal(view, ref)
    del big, view
    torch.cuda.empty_cache()


def test_four_step_batch_of_2_to_the_31():
    """A batch of more than 2^31 elements keeps the tile kernels in both passes."""
    import torch
    need(45)
    torch.cuda.empty_cache()
    n, batch = 1 << 17, (1 << 14) + 2
    x = torch.zeros((batch, n), dtype=torch.complex64, device="cuda")
    rows = [0, 1, 8191, batch - 1]
    cols = columns(len(rows), n, torch.complex64, 5)
    for i, r in enumerate(rows):
        x[r] = cols[i]
    p = F.plan_fft(x.T, 1)
    assert p.describe(x.T).count("[tile") == 2, p.describe(x.T)
    F.mul_(x.T, p, x.T)
    got = torch.stack([x[r] for r in rows])
    assert not x[2:8191:4097].abs().any()
    del x
    torch.cuda.empty_cache()
    ref = np.fft.fft(cols.cpu().numpy().astype(np.complex128))
    err = np.linalg.norm(got.cpu().numpy() - ref) / np.linalg.norm(ref)
    assert err <= 4 * 2.0 ** -23 * np.log2(n)
    assert torch.equal(got, (F.plan_fft(cols.T, 1) * cols.T).T)
