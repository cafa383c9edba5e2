"""The kernels' index arithmetic, checked on the CPU: the reciprocals that
replace divisions (Divisor, fb_internal.h) and the identities behind the
constant shared-memory offsets of a butterfly (Slots, fb_fast.cuh)."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ffta.jl_b200",
                    "csrc")
CUDA = "/usr/local/cuda/include"

DIVISOR = r"""
#include <cstdio>
#include <initializer_list>
#include "fb_internal.h"
int main() {
  const uint32_t top = (1u << 31) - 1;
  for (uint32_t d : {1u, 2u, 3u, 5u, 7u, 9u, 16u, 27u, 243u, 511u, 512u, 513u, 19683u, 65535u,
                     65536u, 65537u, 1048575u, 1073741823u, 1073741824u, 1073741825u, top}) {
    const fb::Divisor q(d);
    if (!q.mul) return std::printf("no reciprocal of %u\n", d), 1;
    for (uint64_t k = 0; k < 4000; ++k)
      for (uint64_t x : {k, k * d, k * d + d - 1, k * d + 1, (uint64_t)top - k, k * 536871u})
        if (x <= top && q.quot((uint32_t)x) != x / d)
          return std::printf("%llu / %u\n", (unsigned long long)x, d), 1;
  }
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="no compiler")
def test_divisor(tmp_path):
    src = tmp_path / "d.cpp"
    src.write_text(DIVISOR)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", f"-I{CUDA}", str(src), "-o",
                    str(tmp_path / "d")], check=True)
    r = subprocess.run([str(tmp_path / "d")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def padi(e):
    return e + (e >> 4)


@pytest.mark.parametrize("radix", [2, 3, 4, 5, 7, 8, 9, 11, 13, 16])
def test_constant_slot_offsets(radix):
    """Where the kernels add r*st + (r*st >> 4) to the first slot of a
    butterfly, that is the slot of element e0 + r*st."""
    for st in range(1, 400):
        step = [r * st + ((r * st) >> 4) for r in range(radix)]
        if st % 16 == 0 or 16 % st == 0:  # reads: e0 = j < st
            assert all(padi(j + r * st) == padi(j) + step[r]
                       for j in range(st) for r in range(radix))
        if st % 16 == 0 or (16 % st == 0 and ((st * radix) % 16 == 0 or 16 % (st * radix) == 0)):
            for m in (0, 1, 2, 3, 17, 100):  # writes: e0 = m*st*radix + k, k < st
                assert all(padi(m * st * radix + k + r * st) == padi(m * st * radix + k) + step[r]
                           for k in range(st) for r in range(radix))
