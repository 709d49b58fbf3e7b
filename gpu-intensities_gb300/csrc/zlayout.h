// How many initial vectors a round takes, and the layout of the half line
// strength Z that follows from the rounds (host arithmetic only).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace gi {

struct FinalSize {  // of a final block
  int ld = 0, nvec = 0;
};
inline FinalSize larger(const FinalSize& a, const FinalSize& b) {
  return FinalSize{std::max(a.ld, b.ld), std::max(a.nvec, b.nvec)};
}
// Workspace bytes of one H column (FP64 and digits) and its column of T.
inline size_t final_col_bytes(const FinalSize& f, size_t digit_bytes) {
  return (size_t)f.ld * (8 + digit_bytes) + (size_t)(f.nvec + (f.nvec & 1)) * 8;
}
// Initial vectors a unit takes: those that fit the workspace, at least one.
inline int unit_vectors(size_t ws_limit, size_t per_vec, size_t nvec) {
  return (int)std::min(std::max<size_t>(1, ws_limit / per_vec), nvec);
}

// Where the elements of a job's Z lie: [3][ncol][ldz], the columns of round
// after round.  In the order of a VibPlan each round pads its column bands to
// whole tiles, so the columns depend on the cut into rounds.
struct ZLayout {
  uint64_t order = 0;        // VibPlan::uid (0: functions as they are, columns unpadded)
  int ldz = 0;
  size_t ncol = 0;
  std::vector<int32_t> cut;  // initial vectors of every round (empty for order 0)
  size_t elems() const { return 3 * ncol * (size_t)ldz; }
  bool operator==(const ZLayout& o) const {
    return order == o.order && ldz == o.ldz && ncol == o.ncol && cut == o.cut;
  }
};

}  // namespace gi
