// ct_range.h -- an INSTANCE's primitive range against the AABB table.  Plain
// C++ for both sides: the kernels that read the ranges before the host has
// checked them, and the host's check.
#pragma once
#include <stdint.h>

#if defined(__CUDACC__)
#define CT_RANGE_FN __host__ __device__ __forceinline__
#else
#define CT_RANGE_FN inline
#endif

// How many of the `count` entries from `first` on lie in a table of n.  The
// entries are first .. first + (the result) - 1, which neither wrap nor pass
// the table's end; fewer than `count` or first > n: the range is outside.
CT_RANGE_FN uint32_t ct_range_inside(uint32_t first, uint32_t count, uint32_t n) {
  const uint32_t left = first < n ? n - first : 0u;
  return count < left ? count : left;
}
CT_RANGE_FN bool ct_range_outside(uint32_t first, uint32_t count, uint32_t n) {
  return first > n || count > n - first;
}
