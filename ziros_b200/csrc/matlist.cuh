// matlist.cuh — the matrices whose rows are concatenated into one leaf.
#pragma once
#include <cstdint>

namespace zkb {

constexpr int MAX_GROUP_MATS = 16;

struct MatList {
  const void *ptr[MAX_GROUP_MATS];
  uint64_t width[MAX_GROUP_MATS];
  uint64_t col_start[MAX_GROUP_MATS + 1];
  int n;
};

template <class F>
__device__ __forceinline__ typename F::T fetch_col(const MatList &ml, uint64_t row, uint64_t col) {
  int m = 0;
  while (m + 1 < ml.n && col >= ml.col_start[m + 1]) m++;
  const typename F::T *base = (const typename F::T *)ml.ptr[m];
  return base[row * ml.width[m] + (col - ml.col_start[m])];
}

}  // namespace zkb
