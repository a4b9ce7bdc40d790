// pq_tc_shape.hpp -- which calls the tensor-core product-quantizer kernel (pq_tc.cu) takes.  Host code only.
#pragma once
#include <cstddef>

namespace vqb {

constexpr size_t PQ_TC_TILE = 128; // rows
// TMA takes the number of a tile's first row as a signed 32-bit coordinate: from row 2^31 on it would be negative, which is no error but
// delivers zeros.
constexpr size_t PQ_TC_MAX_ROWS = size_t(1) << 31;

// Sub-space widths 4 and 8; every number of sub-spaces from four on: the last group of a launch may hold fewer than four, and gets as many
// CTAs as it has work.  Against the CUDA-core kernels (assign_filter.cuh), encode / fit of 5 iterations: 1M rows, 32 of 4: 4.05 -> 0.82 /
// 18.8 -> 5.2 ms; 300,000 rows, 13 of 8: 0.79 -> 0.23 / 4.1 -> 1.6 ms; 100,000 rows, 7 of 4, k 100, cosine: 124 -> 38 us.
inline bool pq_tc_shape(size_t m, size_t sd, size_t k) { return (sd == 4 || sd == 8) && m >= 4 && m <= 64 && k >= 2 && k <= 256; }
inline bool pq_tc_rows(size_t n) { return n >= 1 && n <= PQ_TC_MAX_ROWS; }

} // namespace vqb
