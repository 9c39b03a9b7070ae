// Which pieces of the rows a lane of few_rows_kernel reads: plain arithmetic, apart from the kernel so that a host program
// can walk every shape (tests/test_few_share.py).
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define OMNI_HD __host__ __device__ __forceinline__
#else
#define OMNI_HD inline
#endif

namespace omni {

constexpr int kFewWarps = 8, kFewKb = 64;  // warps of a CTA, K elements of a k-block

// A warp's k-blocks are `per` (the last warps' fewer, or none) of the split's `span`; its lanes stand `lanes` to a row, and a
// piece is eight elements: lane `first` of row n takes pieces first, first + lanes, ... below `pieces`.
struct FewShare {
  int n, first, lanes, pieces, c0;  // c0: the share's first column
  bool live;                        // row n exists
};

OMNI_HD FewShare few_share(int lane, int kb0, int nk, int lanes_log2, int rows) {
  FewShare h;
  h.lanes = 1 << lanes_log2;
  h.n = lane >> lanes_log2, h.first = lane & (h.lanes - 1);
  h.pieces = nk * (kFewKb / 8), h.c0 = kb0 * kFewKb;
  h.live = h.n < rows;
  return h;
}
// Lanes per row (as a power of two): the rows of a warp side by side.
inline int few_lanes_log2(int rows) {
  int log2 = 5;
  while ((32 >> log2) < rows) --log2;
  return log2;
}
// k-blocks per split and per warp.
inline int few_span(int nkb, int splits) { return (nkb + splits - 1) / splits; }
inline int few_per(int nkb, int splits) { return (few_span(nkb, splits) + kFewWarps - 1) / kFewWarps; }
// k-blocks of a warp: the first, and how many there are of it.
OMNI_HD int few_first(int warp, int split, int span, int per) { return split * span + warp * per; }
OMNI_HD int few_count(int warp, int split, int span, int per, int nkb) {
  const int left = nkb - few_first(warp, split, span, per), in_span = span - warp * per;
  const int n = per < in_span ? per : in_span;
  return n < left ? (n < 0 ? 0 : n) : (left < 0 ? 0 : left);
}

// Where a lane's first piece lies in rows of K elements, and its j-th from there. A lane without pieces reads its row's first
// piece of the share with the lane that has it, a warp without k-blocks the rows' first element; what they read is not used.
// (The rows' first element for every idle lane made that line a hot one: a talker step of one session 15 us longer.)
OMNI_HD int64_t few_at(const FewShare& h, int K) {
  return h.pieces > 0 ? (int64_t)(h.live ? h.n : 0) * K + h.c0 + (h.first < h.pieces ? h.first * 8 : 0) : 0;
}
OMNI_HD int few_step(const FewShare& h, int j) { return h.first + j * h.lanes < h.pieces ? j * h.lanes * 8 : 0; }

}  // namespace omni
