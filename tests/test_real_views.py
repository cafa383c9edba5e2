"""Real transforms of torch tensors that are lazily conjugated or negated views:
their storage holds other values than they do."""
import numpy as np
import pytest

import ffta_b200 as F


def test_column_major_memory_holds_the_views_values():
    import torch
    g = torch.Generator().manual_seed(2)
    c = torch.view_as_complex(torch.randn((5, 33, 2), generator=g))
    r = torch.randn((5, 64), generator=g)
    # the imaginary part of a conjugate is the one negated view of real data
    for view in (c.conj().T, torch._neg_view(r).T, c.conj().imag.T, c.T, r.T):
        want = view.clone().resolve_conj().resolve_neg()
        m, dims = F._col_major(view)
        assert dims == tuple(view.shape) and m.is_contiguous()
        assert not m.is_conj() and not m.is_neg()
        raw = np.frombuffer(m.numpy().tobytes(), dtype=m.numpy().dtype).reshape(m.shape)
        assert np.array_equal(raw, want.T.contiguous().numpy())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64, 324])  # one kernel; passes around a complex plan
def test_conjugated_and_negated_views(n):
    import torch
    g = torch.Generator(device="cuda").manual_seed(3)
    x = torch.randn((5, n), generator=g, device="cuda", dtype=torch.float64)
    p = F.plan_rfft(x.T, 1)
    y = p * x.T  # (n/2+1, 5)
    neg = torch._neg_view(x).T
    assert neg.is_neg()
    conj = y.conj()
    assert conj.is_conj()
    q = F.plan_irfft(y, n, 1)
    back = q * conj.resolve_conj()
    straight = q * y
    assert not torch.equal(back, straight)
    for _ in range(2):  # also once a plain array of that layout has been seen
        assert torch.equal(p * neg, p * (-x).T)
        assert torch.equal(q * conj, back)
        assert torch.equal(q * y, straight) and torch.equal(p * x.T, y)
