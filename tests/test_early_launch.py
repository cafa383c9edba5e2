"""Kernels launched while the stream's previous kernel still runs
(launch_overlapped): what that kernel may have written is read by ordinary loads
behind grid_wait, not through the read-only path."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "ffta.jl_b200", "csrc")


def kernels(name):
    """(name, parameters, body) of every __global__ function of a source file."""
    s = open(os.path.join(CSRC, name)).read()
    for m in re.finditer(r"__global__ void\s+(?:__launch_bounds__\([^)]*\)\s+)?(\w+)\(", s):
        depth, i = 1, m.end()
        while depth:  # the parameter list
            depth += {"(": 1, ")": -1}.get(s[i], 0)
            i += 1
        j = s.index("{", i)
        depth, k = 1, j + 1
        while depth:
            depth += {"{": 1, "}": -1}.get(s[k], 0)
            k += 1
        yield m.group(1), s[m.end():i - 1], s[j:k]


def test_helpers_read_their_input_by_ordinary_loads():
    seen = []
    for name, params, body in kernels("fb_kernels.cu"):
        if "grid_wait()" not in body:
            continue
        seen.append(name)
        assert "in" in re.findall(r"\*\s*(?:__restrict__\s+)?(\w+)", params), name
        assert not re.search(r"\*\s*__restrict__\s+(in|out|z)\b", params), name
        after = body[body.index("grid_wait()"):]
        assert not re.search(r"\bin\s*\[|__ldg\(\s*in\b", after), name
        assert re.search(r"__ldc[sa]\(", after), name
    assert {"k_real_to_complex", "k_complex_to_real", "k_extract_half", "k_herm_extend",
            "k_real_half", "k_permute"} <= set(seen)


def test_a_stage_that_loads_and_stores_releases_after_its_loads():
    fast = open(os.path.join(CSRC, "fb_fast.cuh")).read()
    stage = fast[fast.index("void fast_stage("):]
    assert stage.index("row.raw(r)") < stage.index("if constexpr (GOUT) grid_release();")
    line = open(os.path.join(CSRC, "fb_line.cuh")).read()
    stage = line[line.index("void stage("):]
    assert stage.index("finish<RAD>(") < stage.index("if (st) grid_release();")


# one-stage programs in place, the helper directly behind them: neighbouring blocks
# load and store parts of one 32-byte sector
@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("n1,n2", [(63, 7), (255, 7), (101, 3), (45, 16), (2049, 5)])
def test_helpers_behind_one_stage_passes(n1, n2, dtype):
    import torch

    import ffta_b200 as F
    rng = np.random.default_rng(n1 * n2)
    x = torch.from_numpy(rng.standard_normal((n2, n1)).astype(dtype)).cuda()
    p = F.plan_rfft(x.T, (1, 2))
    y = p * x.T
    torch.cuda.synchronize()
    q = F.plan_irfft(y, n1, (1, 2))
    z = q * y
    torch.cuda.synchronize()
    ref = np.fft.fft(np.fft.rfft(x.cpu().numpy().astype(np.float64), axis=1), axis=0)
    eps = np.finfo(dtype).eps
    bound = 4 * eps * np.log2(n1 * n2)
    assert np.linalg.norm(y.T.cpu().numpy() - ref) <= bound * np.linalg.norm(ref)
    a, b = [], []
    for _ in range(64):  # back to back, every launch close behind the last
        a.append(p * x.T)
        b.append(q * a[-1])
    torch.cuda.synchronize()
    assert all(torch.equal(v, y) for v in a) and all(torch.equal(v, z) for v in b)


@pytest.mark.gpu
def test_tables_made_by_the_previous_kernel():
    """fb_execute_noalloc_c32 writes its tables on the stream of each call:
    alternating lengths, the same bits as each alone."""
    import ctypes

    import torch
    from ffta_b200 import _lib
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(1)
    xs = [torch.view_as_complex(torch.randn((3, n, 2), generator=g, device="cuda"))
          for n in (960, 4096, 45000)]

    def run(x):
        y = torch.empty_like(x)
        rc = _lib.lib.fb_execute_noalloc_c32(ctypes.c_void_p(x.data_ptr()),
                                             ctypes.c_void_p(y.data_ptr()), x.shape[1], x.shape[0],
                                             -1, stream)
        assert rc == _lib.FB_OK, _lib.last_error()
        return y

    alone = []
    for x in xs:
        alone.append(run(x))
        torch.cuda.synchronize()
        ref = np.fft.fft(x.cpu().numpy().astype(np.complex128))
        err = np.linalg.norm(alone[-1].cpu().numpy() - ref) / np.linalg.norm(ref)
        assert err <= 4 * 2.0 ** -23 * np.log2(x.shape[1])
    out = [[run(x) for x in xs] for _ in range(20)]
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for row in out for a, b in zip(row, alone))
