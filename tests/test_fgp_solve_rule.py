"""The rule that picks the FGP kernel of a solve (fgp_solve_cost in fgp_rule.h),
compiled alone with the host compiler, against measured TV solves with every
candidate on B200 (FGP 50, a lambda grid): (FP64, pixels a side, problems,
[(rows a thread, CTAs a problem, problems resident at once, milliseconds of 100
iterations, of up to 300 to eps 1e-4)])."""
import os
import subprocess

import pytest

from conftest import ROOT

MEASURED = [
    (1, 64, 24, [(0, 16, 31, 35, 93), (0, 8, 71, 40, 112), (1, 16, 31, 27, 70), (1, 8, 33, 28, 76), (2, 16, 66, 37, 101), (2, 8, 71, 38, 105)]),
    (1, 72, 16, [(0, 16, 31, 39, 107), (0, 8, 71, 45, 127), (1, 16, 14, 27, 70), (1, 8, 15, 28, 70), (2, 16, 31, 38, 104), (2, 8, 33, 37, 99)]),
    (1, 72, 64, [(0, 16, 31, 74, 158), (0, 8, 71, 56, 148), (1, 16, 14, 67, 142), (1, 8, 15, 66, 138), (2, 16, 31, 72, 154), (2, 8, 33, 69, 140)]),
    (1, 96, 8, [(0, 16, 31, 45, 133), (0, 8, 71, 65, 183), (1, 16, 7, 27, 68), (2, 16, 21, 36, 96), (2, 8, 15, 40, 109)]),
    (1, 96, 16, [(0, 16, 31, 50, 133), (0, 8, 71, 107, 191), (1, 16, 7, 42, 84), (2, 16, 21, 43, 113), (2, 8, 15, 52, 114)]),
    (1, 96, 24, [(0, 16, 31, 52, 136), (0, 8, 71, 70, 197), (1, 16, 7, 53, 121), (2, 16, 21, 46, 117), (2, 8, 15, 71, 137)]),
    (1, 96, 64, [(0, 16, 31, 93, 197), (0, 8, 71, 80, 218), (1, 16, 7, 114, 241), (2, 16, 21, 100, 222), (2, 8, 15, 119, 252)]),
    (1, 128, 8, [(0, 16, 31, 54, 151), (0, 8, 33, 81, 229), (1, 16, 7, 31, 79), (2, 16, 14, 59, 122), (2, 8, 15, 47, 128)]),
    (1, 128, 16, [(0, 16, 31, 59, 156), (0, 8, 33, 83, 233), (1, 16, 7, 47, 96), (2, 16, 14, 47, 124), (2, 8, 15, 50, 132)]),
    (1, 128, 64, [(0, 16, 31, 111, 232), (0, 8, 33, 148, 313), (1, 16, 7, 121, 257), (2, 16, 14, 129, 275), (2, 8, 15, 139, 292)]),
    (1, 144, 16, [(0, 16, 21, 93, 264), (0, 8, 15, 152, 439), (2, 16, 7, 71, 149)]),
    (1, 160, 24, [(0, 16, 21, 106, 294), (0, 8, 15, 266, 583), (2, 16, 7, 99, 217)]),
    (0, 64, 64, [(0, 16, 45, 65, 150), (0, 8, 104, 58, 152), (1, 16, 31, 55, 111), (1, 8, 33, 53, 113), (2, 16, 66, 50, 128), (2, 8, 71, 55, 131)]),
    (0, 72, 16, [(0, 16, 45, 50, 135), (0, 8, 104, 58, 161), (1, 16, 14, 35, 90), (1, 8, 15, 35, 90), (2, 16, 31, 44, 120), (2, 8, 33, 44, 120)]),
    (0, 96, 8, [(0, 16, 45, 57, 158), (0, 8, 104, 84, 240), (1, 16, 7, 34, 87), (2, 16, 21, 44, 119), (2, 8, 15, 46, 125)]),
    (0, 96, 24, [(0, 16, 45, 66, 173), (0, 8, 104, 89, 250), (1, 16, 7, 65, 150), (2, 16, 21, 51, 131), (2, 8, 15, 69, 151)]),
    (0, 128, 16, [(0, 16, 45, 74, 203), (0, 8, 71, 107, 301), (1, 16, 7, 54, 118), (2, 16, 14, 53, 137), (2, 8, 15, 57, 148)]),
    (0, 128, 64, [(0, 16, 45, 122, 310), (0, 8, 71, 130, 360), (1, 16, 7, 143, 305), (2, 16, 14, 133, 292), (2, 8, 15, 134, 295)]),
    (0, 144, 24, [(0, 16, 45, 123, 344), (0, 8, 48, 195, 569), (2, 16, 7, 96, 221)]),
    (0, 160, 8, [(0, 16, 38, 126, 361), (0, 8, 48, 213, 627), (2, 16, 7, 54, 143)]),
    (0, 160, 24, [(0, 16, 38, 138, 380), (0, 8, 48, 220, 640), (2, 16, 7, 101, 228)]),
]

DRIVER = r"""
#include "fgp_rule.h"
#include <cstdio>
int main() {
  int fp64, n, b, nr, cs, resident;
  while (scanf("%d %d %d %d %d %d", &fp64, &n, &b, &nr, &cs, &resident) == 6)
    printf("%.17g\n", mf::fgp_solve_cost(mf::FgpCandidate{nr, cs, resident}, fp64 != 0, n, n, b, 148));
  return 0;
}
"""


@pytest.fixture(scope="module")
def cost(tmp_path_factory):
    d = tmp_path_factory.mktemp("fgp")
    (d / "rule.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "sparseimaging_b200", "csrc"), "-o",
                    str(d / "rule"), str(d / "rule.cpp")], check=True)

    def call(rows):
        text = "\n".join(" ".join(str(v) for v in r) for r in rows)
        out = subprocess.run([str(d / "rule")], input=text, capture_output=True, text=True, check=True).stdout
        return [float(v) for v in out.split()]
    return call


@pytest.mark.parametrize("fp64, n, b, candidates", MEASURED)
def test_pick_is_among_the_fastest(cost, fp64, n, b, candidates):
    """The mean of the two solves, each against its fastest candidate: within
    15 % (the rule's worst is 10 %)."""
    c = cost([(fp64, n, b, nr, cs, res) for nr, cs, res, *_ in candidates])
    pick = candidates[c.index(min(c))]
    over = [pick[k] / min(t[k] for t in candidates) for k in (3, 4)]
    assert sum(over) / 2 <= 1.15
