"""Rules on the kernels' sources that no run can show broken."""
import os
import re
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "f3r_b200", "csrc")
# what no kernel of a stream writes: a matrix's values, columns, slot bases and row patterns
CONSTANT = re.compile(r"^(val|ival|tab)$|^(lc|lv)\b|^(reinterpret_cast<const int4 \*>\()?\(?A\.")


def _sources():
    for f in sorted(os.listdir(CSRC)):
        if f.endswith((".cuh", ".cu")):
            with open(os.path.join(CSRC, f)) as s:
                yield f, s.read()


def test_kernels_that_may_start_early_read_results_coherently():
    """A kernel that begins with stream_order() may be resident while its
    predecessor still writes: it takes no read-only path (const __restrict__,
    __ldg) to anything but constants of the matrix."""
    kernels = 0
    for f, s in _sources():
        early = list(re.finditer(r"__global__[^{;]*?(k_\w+)\(([^{;]*)\)\s*\{\n  stream_order\(\);", s))
        kernels += len(early)
        for m in early:
            for p in re.findall(r"__restrict__\s+(\w+)", m.group(2)):
                assert CONSTANT.match(p), (f, m.group(1), p)
        if early and f not in ("block.cuh", "kernels.cuh"):  # these two hold kernels that never start early, too
            for a in re.findall(r"__ldg\((.*)", s):
                assert CONSTANT.match(a), (f, a)
    assert kernels >= 15


def test_rows_off_the_patterns_are_dealt_evenly(tmp_path):
    """every round to one CTA, and no CTA with more than its share of tiles and
    rounds (a tile as kRestSpare rounds) and one of each, whatever the last wave holds"""
    src = tmp_path / "rest.cpp"
    src.write_text(r'''
#include <cstdio>
#include <vector>
#include "patrest.hpp"
using namespace f3r;
int main() {
  for (int grid : {1, 2, 147, 148, 296, 444, 592})
    for (int tiles : {0, 1, 146, 147, 148, 295, 442, 443, 444, 583, 1175, 2662, 3456})
      for (int groups : {0, 1, 7, 8, 9, 985, 2058, 4000, 16815, 400000}) {
        const PatRest r(tiles, groups, 8, grid);
        std::vector<int> seen(r.rounds, 0);
        const double share = (tiles * (double)kRestSpare + r.rounds) / grid;
        for (int c = 0; c < grid; c++) {
          int mine = 0;
          for (int q = r.begin(c, grid); q < r.rounds; q = r.next(q, c, grid), mine++) seen[q]++;
          const int t = c < tiles ? (tiles - 1 - c) / grid + 1 : 0;
          const double load = t * (double)kRestSpare + mine;
          if (mine && load > share + kRestSpare + 1) return std::printf("%d %d %d: CTA %d %d + %d\\n", grid, tiles, groups, c, t, mine), 1;
        }
        for (int k : seen)
          if (k != 1) return std::printf("%d %d %d: a round dealt %d times\\n", grid, tiles, groups, k), 1;
        if (r.rounds * 8 < groups || (r.rounds - 1) * 8 >= groups + 8) return 1;
      }
  return 0;
}
''')
    exe = tmp_path / "rest"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
