"""The shared-memory slots of the kernels' butterflies (fb_internal.h), the
functions themselves compiled for the host: the constant offsets of the compiled
kernels (const_slots, slot_step) and the generic kernel's form (GenSlots) against
slot_of, element by element."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ffta.jl_b200",
                    "csrc")
CUDA = "/usr/local/cuda/include"

SLOTS = r"""
#include <cstdio>
#include <initializer_list>
#include "fb_internal.h"
using namespace fb;
int main() {
  long taken = 0;
  for (bool flat : {false, true})
    for (int rad : {2, 3, 4, 5, 7, 8, 9, 11, 13, 16})
      for (int st = 1; st < 700; ++st) {
        if (const_slots(flat, rad, st, false))  // reads: e0 = j < st
          for (int j = 0; j < st; ++j)
            for (int r = 0; r < rad; ++r, ++taken)
              if (slot_of(flat, j + r * st) != slot_of(flat, j) + slot_step(flat, r * st))
                return std::printf("read %d %d %d %d\n", rad, st, j, r), 1;
        if (const_slots(flat, rad, st, true))  // writes: e0 = m*st*rad + k, k < st
          for (int m : {0, 1, 2, 3, 5, 17, 100})
            for (int k = 0; k < st; ++k)
              for (int r = 0; r < rad; ++r, ++taken)
                if (slot_of(flat, m * st * rad + k + r * st) !=
                    slot_of(flat, m * st * rad + k) + slot_step(flat, r * st))
                  return std::printf("write %d %d %d %d %d\n", rad, st, m, k, r), 1;
        for (int e = 0; e < 40; ++e) {
          const GenSlots g(e * 37, st);
          for (int r = 0; r < rad; ++r)
            if (g[r] != slot_of(false, e * 37 + r * st))
              return std::printf("generic %d %d %d\n", e * 37, st, r), 1;
        }
      }
  // strides that the compiled programs meet take the constant form
  for (int st : {1, 2, 4, 8, 16, 64, 256, 512})
    if (!const_slots(false, 16, st, false) || !const_slots(false, 16, st, true)) return 1;
  if (const_slots(false, 9, 3, false) || const_slots(false, 3, 2, true)) return 1;
  // no two elements of a line share a slot
  for (int e = 0; e < 20000; ++e)
    if (slot_of(false, e + 1) <= slot_of(false, e) || slot_of(true, e) != e) return 1;
  return taken > 100000 ? 0 : 1;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA), reason="no compiler")
def test_slots(tmp_path):
    src = tmp_path / "s.cpp"
    src.write_text(SLOTS)
    subprocess.run(["g++", "-std=c++17", "-O1", f"-I{CSRC}", f"-I{CUDA}", str(src), "-o",
                    str(tmp_path / "s")], check=True)
    r = subprocess.run([str(tmp_path / "s")], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
