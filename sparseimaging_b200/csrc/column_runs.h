// Which columns of a host matrix go to the device, and in how many copies.
#pragma once
#include <cstddef>
#include <vector>

namespace mf {

struct ColumnRun {
  int first, last;  // columns [first, last)
};

// A copy from pageable memory costs 11 us and 11.4 GB/s on B200 (4 KB 7 us,
// 64 KB 17 us, 1 MB 116 us), as much as 128 KB more in a copy that is under
// way.  Pinned memory (53 GB/s) would stand 0.5 MB; columns copied along cost
// it at most 2.5 us a run.
constexpr size_t kColumnGapBytes = 128 * 1024;

// The used columns in runs of neighbours; a run takes unused columns along
// where they are fewer bytes than another copy costs.
inline std::vector<ColumnRun> column_runs(const std::vector<char>& used, size_t column_bytes) {
  std::vector<ColumnRun> runs;
  for (int j = 0; j < (int)used.size(); ++j) {
    if (!used[j]) continue;
    if (!runs.empty() && (size_t)(j - runs.back().last) * column_bytes <= kColumnGapBytes)
      runs.back().last = j + 1;
    else
      runs.push_back(ColumnRun{j, j + 1});
  }
  return runs;
}

}  // namespace mf
