"""The transforms whose speed is followed: planned FFTs on device-resident data.

A case is a plan kept by the program (`plan_fft`, `plan_bfft`, `plan_ifft`,
`plan_rfft`, `plan_irfft`) applied once to one array: `mul_(y, p, x)` for
complex transforms, `p * x` for real ones.  Arrays are in Julia's column-major
order: `dims` are the transformed dimensions, first one contiguous, and
`batch` independent transforms follow one another in memory.

The listed cases are the shapes of this repository's benchmark (one small
transform; batches of powers of two and three, of mixed lengths, of
composites and of primes; images; real transforms).  `draw` spreads over the
ranges behind them: lengths from 16 to 2^20 of every factorisation class, the
class mix and the share of ComplexF32 of the serving stream, batches from one
transform to the largest listed array, both directions.
"""
import math
import os
import sys
from functools import lru_cache

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "ffta.jl_b200"))

import ffta_b200 as F  # noqa: E402

_REAL = {"f32": torch.float32, "f64": torch.float64}
_CPLX = {"f32": torch.complex64, "f64": torch.complex128}


def _case(name, op, prec, dims, batch):
    n1, n2 = (tuple(dims) + (1,))[:2]
    c = {"op": op, "prec": prec, "rank": len(dims), "n1": n1, "n2": n2, "batch": batch}
    return dict(c, name=name) if name else c


def listed():
    return [
        # one small transform: call overhead and one short kernel
        _case("one_1024_f64", "fft", "f64", (1024,), 1),
        # the headline batch of short columns, both inputs and outputs beyond L2
        _case("columns_4096_f32", "fft", "f32", (4096,), 16384),
        # the same length in double precision, the unnormalised inverse
        _case("columns_4096_f64", "bfft", "f64", (4096,), 4096),
        # powers of three in double precision, scaled inverse: long columns
        _case("columns_19683_f64", "ifft", "f64", (19683,), 852),
        # 2^10 * 3^3: mixed radices, a ragged number of columns
        _case("columns_27648_f32", "bfft", "f32", (27648,), 606),
        # long transforms: several passes over memory
        _case("long_1048576_f32", "fft", "f32", (1 << 20,), 16),
        # a composite with factors 5, 7 and 11
        _case("composite_23100_f32", "fft", "f32", (23100,), 256),
        # a prime length (Bluestein), a few transforms
        _case("prime_65537_f32", "fft", "f32", (65537,), 16),
        # a large image, forward
        _case("image_4096x4096_f32", "fft", "f32", (4096, 4096), 1),
        # an ordinary image with factors of five, scaled inverse
        _case("image_1000x1000_f32", "ifft", "f32", (1000, 1000), 1),
        # real signals to half spectra
        _case("real_4096_f32", "rfft", "f32", (4096,), 16384),
        # half spectra of a real image in double precision back to the image
        _case("real_image_1000x1000_f64", "irfft", "f64", (1000, 1000), 1),
    ]


# ------------------------------------------------------------------- drawing
def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _rest(n, primes):
    """What is left of n once these primes are divided out."""
    for p in primes:
        while n % p == 0:
            n //= p
    return n


def _length(rng, lo, hi, primes=True):
    """A length in lo..hi of the stream's class mix: 50% powers of two, 20%
    2^a 3^b, 15% other smooth numbers, 15% primes (or smooth, without them)."""
    k = rng.random()
    if k < 0.5:
        return 1 << rng.randint(math.ceil(math.log2(lo)), int(math.log2(hi)))
    n = int(_log_uniform(rng, lo, hi))
    if k < 0.7:
        fits = lambda m: m % 3 == 0 and _rest(m, (2, 3)) == 1  # noqa: E731
    elif k < 0.85 or not primes:
        fits = lambda m: _rest(m, (2, 3)) > 1 and _rest(m, (2, 3, 5, 7, 11, 13)) == 1  # noqa: E731
    else:
        fits = lambda m: m > 1 and all(m % d for d in range(2, math.isqrt(m) + 1))  # noqa: E731
    while n > lo and not fits(n):
        n -= 1
    return n


def _cap(n):
    """Elements of one array at most: the listed cases' sizes, by class."""
    if _rest(n, (2, 3)) == 1:
        return 1 << 24
    return 23100 * 256 if _rest(n, (2, 3, 5, 7, 11, 13)) == 1 else 1 << 20


def draw(rng):
    kind = rng.random()
    prec = "f32" if rng.random() < 0.8 else "f64"
    wide = 1 if prec == "f32" else 2
    if kind < 0.6:  # batched columns
        dims = (_length(rng, 16, 1 << 20),)
        op = rng.choice(("fft", "bfft", "ifft"))
    elif kind < 0.75:  # images
        dims = tuple(_length(rng, 32, 4096, primes=False) for _ in range(2))
        op = rng.choice(("fft", "bfft", "ifft"))
    elif kind < 0.9:  # real columns, even and odd lengths
        dims = (_length(rng, 16, 1 << 18),)
        op = rng.choice(("rfft", "irfft"))
    else:  # real images
        dims = tuple(_length(rng, 32, 2048, primes=False) for _ in range(2))
        op = rng.choice(("rfft", "irfft"))
    n = math.prod(dims)
    most = max(1, min(_cap(d) for d in dims) // (wide * n))
    return _case("", op, prec, dims, int(_log_uniform(rng, 1, most + 1)))


# ------------------------------------------------------------------- running
def _dims(case):
    return (case["n1"], case["n2"])[: case["rank"]]


def _memory_shape(case, half=False):
    """Shape of the array as it lies in memory, last axis contiguous."""
    d = list(_dims(case))
    if half:
        d[0] = d[0] // 2 + 1
    return (case["batch"], *reversed(d))


def _julia(t):
    """The column-major view of a contiguous tensor, as Julia sees it."""
    return t.permute(tuple(range(t.ndim - 1, -1, -1)))


def _input(case, seed):
    """The input as it lies in memory: i.i.d. normal samples (sigma 1 per
    part), or for the inverse real transform the half spectrum of such."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = _memory_shape(case)
    if case["op"] in ("rfft", "irfft"):
        x = torch.randn(shape, dtype=_REAL[case["prec"]], device="cuda", generator=g)
        if case["op"] == "rfft":
            return x
        axes = tuple(range(-1, -1 - case["rank"], -1))
        return torch.fft.rfftn(x, dim=tuple(reversed(axes))).contiguous()
    parts = torch.randn(shape + (2,), dtype=_REAL[case["prec"]], device="cuda", generator=g)
    return torch.view_as_complex(parts)


# one plan serves every array of a shape, as in a program that transforms
# many of them
@lru_cache(maxsize=1)
def _plan(op, prec, rank, n1, n2, batch):
    case = {"rank": rank, "n1": n1, "n2": n2, "batch": batch}
    region = tuple(range(1, rank + 1))
    half = op == "irfft"
    dtype = _REAL[prec] if op == "rfft" else _CPLX[prec]
    x = _julia(torch.empty(_memory_shape(case, half), dtype=dtype, device="cuda"))
    if op == "irfft":
        return F.plan_irfft(x, n1, region)
    plan = {"fft": F.plan_fft, "bfft": F.plan_bfft, "ifft": F.plan_ifft, "rfft": F.plan_rfft}
    return plan[op](x, region)


def prepare(case, seed):
    keys = ("op", "prec", "rank", "n1", "n2", "batch")
    t = _input(case, seed)
    state = {"plan": _plan(*(case[k] for k in keys)), "x": _julia(t)}
    if not case["op"].endswith("rfft"):
        state["out"] = torch.empty_like(t)
        state["y"] = _julia(state["out"])
    return state


def run(state):
    if "y" in state:
        F.mul_(state["y"], state["plan"], state["x"])
        return state["out"]
    return _julia(state["plan"] * state["x"])


def work(case):
    es = 8 if case["prec"] == "f32" else 16
    n = math.prod(_memory_shape(case))
    flops = 5.0 * n * math.log2(math.prod(_dims(case)))
    if not case["op"].endswith("rfft"):
        return {"bytes": 2 * n * es, "flops": flops}
    half = math.prod(_memory_shape(case, half=True))
    return {"bytes": n * es // 2 + half * es, "flops": flops / 2}


def exact(case, seed):
    x = _input(case, seed).cpu().numpy()
    axes = tuple(range(-case["rank"], 0))
    if case["op"] == "rfft":
        return np.fft.rfftn(x.astype(np.float64), axes=axes)
    x = x.astype(np.complex128)
    if case["op"] == "fft":
        return np.fft.fftn(x, axes=axes)
    if case["op"] == "bfft":
        return np.fft.ifftn(x, axes=axes, norm="forward")
    if case["op"] == "ifft":
        return np.fft.ifftn(x, axes=axes)
    shape = tuple(reversed(_dims(case)))
    return np.fft.irfftn(x, s=shape, axes=axes)
