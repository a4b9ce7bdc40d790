// queue_sums.cuh -- cluster sums in no particular order (queue_sums.cu).
#pragma once
#include <cstddef>
#include <cstdint>

namespace vqb {

class CudaDevice;
struct Shape;

// one-byte codes, sub-spaces of 4 to 32 dimensions (moved rows: 128) in whole 16-byte pieces
bool queue_sums_applicable(CudaDevice &dev, const Shape &sh, const float *x, const float *sums, size_t code_bytes, bool moved);

// codes_prev == nullptr: adds every row to the sums and counts of its clusters.  Otherwise only the rows whose code differs
// from codes_prev are moved from the old cluster to the new one, and codes_prev is brought up to date.
void launch_queue_sums(CudaDevice &dev, const Shape &sh, const float *x, uint8_t *codes_prev, const uint8_t *codes, const uint32_t *active, float *sums,
                       uint32_t *counts, bool counts_f32);

} // namespace vqb
