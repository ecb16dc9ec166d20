"""Rules on the kernels' sources that no run can show broken."""
import os
import re

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
