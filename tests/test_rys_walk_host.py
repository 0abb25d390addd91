"""The walk of a launch's quartets in the Rys-quadrature kernels (rys_first, rys_stride and rys_blocks of
csrc/hfgpu_rys_math.cuh), compiled with g++ and run on the host at list lengths around 2^30 and 2^31 - 1,
where a 32-bit index overflows in its first step.

Every index a walker reaches is inside the list, the walkers of consecutive blocks tile it without a gap
or an overlap, and a walk ends.  Exact whole numbers.
"""
import os
import re
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "hfscf_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include <initializer_list>
#define __host__
#define __device__
#include "walk.h"
#define CHECK(x) if (!(x)) { std::printf("%s: nq %lld walkers %d per %d most %d\n", #x, nq, walkers, per, most); return 1; }
int main() {
  for (long long nq : {1ll, 19ll, 20ll, 21ll, (1ll << 30) - 1, 1ll << 30, (1ll << 30) + 1, (1ll << 31) - 40, (1ll << 31) - 1})
    for (int walkers : {1, 2, 4})
      for (int per : {1, 2, 10, 20, 64})
        for (int most : {0, 148, 2048}) {
          const unsigned blocks = rys_blocks(nq, walkers, per, most);
          const long long turn = rys_stride(blocks, walkers, per);
          CHECK(blocks > 0 && (most == 0 || blocks <= (unsigned)most));
          CHECK(most > 0 || (turn >= nq && turn - (long long)walkers * per < nq));
          CHECK(rys_first(0, walkers, 0, per) == 0);
          for (unsigned b : {0u, blocks / 2, blocks - 1}) {
            for (int w = 0; w < walkers; ++w) {
              // the next walker, or the first one's next turn, takes over where this one ends
              const long long end = rys_first(b, walkers, w, per) + per;
              const long long next = w + 1 < walkers ? rys_first(b, walkers, w + 1, per)
                                     : (b + 1 < blocks ? rys_first(b + 1, walkers, 0, per) : turn);
              CHECK(end == next);
            }
            long long turns = 0;
            for (long long q = rys_first(b, walkers, 0, per); q < nq; q += rys_stride(blocks, walkers, per)) {
              CHECK(q >= 0 && ++turns <= nq / turn + 1);
            }
          }
        }
  return 0;
}
"""


def test_quartet_walk_in_64_bits(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("g++ not available")
    text = open(os.path.join(CSRC, "hfgpu_rys_math.cuh")).read()
    fns = re.findall(r"__host__ __device__ constexpr \w+(?: \w+)? rys_(?:first|stride|blocks)\(.*?\n}\n", text, re.S)
    assert len(fns) == 3
    (tmp_path / "walk.h").write_text("\n".join(fns))
    (tmp_path / "walk.cpp").write_text(DRIVER)
    exe = tmp_path / "walk"
    subprocess.run([gxx, "-std=c++17", "-O1", "-fsanitize=undefined", "-fno-sanitize-recover", "-I", str(tmp_path),
                    str(tmp_path / "walk.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("name", ["hfgpu_rys.cuh", "hfgpu_rys3.cuh", "hfgpu_rys_jk.cuh"])
def test_the_kernels_walk_by_these_functions(name):
    text = open(os.path.join(CSRC, name)).read()
    loops = re.findall(r"for \(([\w ]+) (?:q0|qi) = (\w+)\(.*?; \w+ < nq; \w+ \+= (\w+)\(", text)
    assert loops == [("long long", "rys_first", "rys_stride")]
