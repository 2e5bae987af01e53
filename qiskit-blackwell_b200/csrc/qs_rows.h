// qs_rows.h — one lane's way through the entries of a CSR row.
//
// Row pointers are int32, so a row may end at 2^31 - 1 and a lane that looks
// some entries ahead must not add to its position in 32 bits: the walk counts
// what is left of the row, and the position is 64 bits wide.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define QS_ROWS_HD __host__ __device__ __forceinline__
#else
#define QS_ROWS_HD inline
#endif

struct RowWalk {
  int64_t at;     // the lane's next entry
  int32_t left;   // entries from there to the end of the row (may be negative)
  QS_ROWS_HD RowWalk(int32_t begin, int32_t end, int lane)
      : at((int64_t)begin + lane), left(end - begin - lane) {}
  QS_ROWS_HD bool more() const { return left > 0; }
  QS_ROWS_HD bool has(int ahead) const { return ahead < left; }
  QS_ROWS_HD void step(int n) {
    at += n;
    left -= n;
  }
};
