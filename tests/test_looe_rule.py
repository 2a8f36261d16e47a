"""On how many streams the leave-one-out errors of a call run (looe_rule.h),
compiled alone with the host compiler: further streams only where the solutions
they take pay for them, never more than solutions or than asked for."""
import os
import subprocess

import pytest

from conftest import ROOT

DRIVER = r"""
#include "looe_rule.h"
#include <cstdio>
int main() {
  int b, p, rows, most;
  while (scanf("%d %d %d %d", &b, &p, &rows, &most) == 4) printf("%d\n", mf::looe_lanes(b, p, rows, most));
  return 0;
}
"""


@pytest.fixture(scope="module")
def lanes(tmp_path_factory):
    d = tmp_path_factory.mktemp("lanes")
    (d / "lanes.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "sparseimaging_b200", "csrc"), "-o",
                    str(d / "lanes"), str(d / "lanes.cpp")], check=True)

    def call(cases):
        out = subprocess.run([str(d / "lanes")], input="\n".join("%d %d %d %d" % c for c in cases), capture_output=True,
                             text=True, check=True).stdout
        return [int(x) for x in out.split()]
    return call


def test_bounds(lanes):
    cases = [(b, p, m, most) for b in (0, 1, 2, 3, 4, 5, 7, 64, 10000) for p in (0, 1, 2, 20, 1025, 1 << 20)
             for m in (1, 8000, 1 << 30) for most in (1, 2, 4)]
    for (b, _, _, most), n in zip(cases, lanes(cases)):
        assert 1 <= n <= max(1, min(b, most))


def test_few_small_solutions_share_a_stream(lanes):
    """Two or three solutions of up to 64 pixels and few rows: a call on two or
    three streams took 5-15 % longer than on one."""
    assert lanes([(2, 1, 40, 4), (3, 1, 40, 4), (3, 1, 100, 4)]) == [1, 1, 1]


def test_large_or_many_solutions_do_not(lanes):
    assert lanes([(3, 20, 8000, 4), (4, 20, 8000, 4), (64, 20, 40, 4), (64, 1, 40, 4), (3, 1, 3000, 4)]) == [3, 4, 4, 4, 3]
