"""The copies of a host matrix's used columns (column_runs.h), compiled alone
with the host compiler: every used column is in exactly one run, and runs part
only where the columns between them are more bytes than another copy costs."""
import os
import subprocess

import numpy as np
import pytest

from conftest import ROOT

DRIVER = r"""
#include "column_runs.h"
#include <cstdio>
int main() {
  int n;
  size_t bytes;
  if (scanf("%d %zu", &n, &bytes) != 2) return 1;
  std::vector<char> used(n);
  for (char& u : used) {
    int v;
    if (scanf("%d", &v) != 1) return 1;
    u = (char)v;
  }
  printf("%zu", mf::kColumnGapBytes);
  for (const mf::ColumnRun& r : mf::column_runs(used, bytes)) printf(" %d %d", r.first, r.last);
  return 0;
}
"""


@pytest.fixture(scope="module")
def runs(tmp_path_factory):
    d = tmp_path_factory.mktemp("runs")
    (d / "runs.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I" + os.path.join(ROOT, "sparseimaging_b200", "csrc"), "-o",
                    str(d / "runs"), str(d / "runs.cpp")], check=True)

    def call(used, column_bytes):
        text = f"{len(used)} {column_bytes}\n" + " ".join(str(int(u)) for u in used)
        out = subprocess.run([str(d / "runs")], input=text, capture_output=True, text=True, check=True).stdout.split()
        v = [int(x) for x in out]
        return v[0], [tuple(v[i:i + 2]) for i in range(1, len(v), 2)]
    return call


@pytest.mark.parametrize("m", [2, 20, 300, 3000, 8000, 40000])
@pytest.mark.parametrize("n, active", [(4096, 400), (4096, 1), (64, 64), (1, 1), (5000, 20), (16384, 0)])
def test_runs_cover_the_used_columns(runs, m, n, active):
    rng = np.random.default_rng(n + active)
    used = np.zeros(n, bool)
    used[rng.choice(n, active, replace=False)] = True
    gap, r = runs(used, 8 * m)
    covered = np.zeros(n, int)
    for a, b in r:
        assert used[a] and used[b - 1]
        covered[a:b] += 1
    assert covered.max(initial=0) <= 1 and (covered[used] == 1).all()
    for (_, b), (a, _) in zip(r, r[1:]):
        assert (a - b) * 8 * m > gap


def test_few_rows_are_one_copy(runs):
    """400 scattered columns of 300 rows (2.4 KB each): a handful of copies, not
    one for every used column."""
    used = np.zeros(4096, bool)
    used[np.random.default_rng(0).choice(4096, 400, replace=False)] = True
    assert len(runs(used, 8 * 300)[1]) <= 4
