"""The box of quads whose sectors the backprojector loads ahead of its samples (csrc/footprint.cuh, the
function the kernels call, compiled for the host): it has to lie inside the view for any corners, because the
loads are real ones.  Corners at the source project to infinity, which converts to the ends of int; every
operation is checked for signed overflow (-fsanitize=signed-integer-overflow aborts on one)."""
import itertools
import subprocess
from pathlib import Path

import numpy as np
import pytest

CSRC = Path(__file__).resolve().parent.parent / "listctrecons_b200" / "csrc"

PROGRAM = r"""
#include <cstdio>
#include "footprint.cuh"
int main() {
  int ns, nt;
  int4 c;
  while (std::scanf("%d %d %d %d %d %d", &ns, &nt, &c.x, &c.y, &c.z, &c.w) == 6) {
    const int4 b = lct::box_in_view(c, ns, nt);
    std::printf("%d %d %d %d\n", b.x, b.y, b.z, b.w);
  }
}
"""


@pytest.fixture(scope="module")
def boxes(tmp_path_factory):
    d = tmp_path_factory.mktemp("footprint")
    (d / "box.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-fsanitize=signed-integer-overflow",
                    "-fno-sanitize-recover=all", "-I", str(CSRC), "-I", "/usr/local/cuda/include",
                    str(d / "box.cpp"), "-o", str(d / "box")], check=True)

    def run(rows):
        text = "\n".join(" ".join(str(int(v)) for v in r) for r in rows)
        out = subprocess.run([str(d / "box")], input=text, capture_output=True, text=True, check=True)
        return np.array([[int(v) for v in line.split()] for line in out.stdout.splitlines()])

    return run


def test_box_lies_inside_the_view_for_any_corners(boxes):
    lo, hi = -2 ** 31, 2 ** 31 - 1
    ends = [lo, lo + 1, lo + 2, -4, -1, 0, 1, 5, 8, 9, 10, 11, 12, hi - 3, hi - 2, hi - 1, hi]
    rows = [(9, 7, *c) for c in itertools.product(ends, repeat=4) if c[0] <= c[1] and c[2] <= c[3]]
    rows += [(1, 1, *c) for c in itertools.product((lo, 0, 1, hi), repeat=4)]
    got = boxes(rows)
    assert len(got) == len(rows)
    r = np.array(rows, dtype=np.int64)
    ns, nt = r[:, 0], r[:, 1]
    x = np.minimum(np.maximum(r[:, 2] - 1, 0), nt + 2)
    y = np.minimum(np.maximum(r[:, 3] + 1, x), nt + 2)
    z = np.minimum(np.maximum(r[:, 4] + 1, 0), ns + 2)
    w = np.minimum(np.maximum(r[:, 5] + 3, z), ns + 2)
    assert np.array_equal(got, np.stack([x, y, z, w], axis=1))
    assert (got[:, 0] >= 0).all() and (got[:, 0] <= got[:, 1]).all() and (got[:, 1] <= nt + 2).all()
    assert (got[:, 2] >= 0).all() and (got[:, 2] <= got[:, 3]).all() and (got[:, 3] <= ns + 2).all()
