// ordered_sums.cuh -- cluster sums in ascending row order (the serial branch of mean_vector, src/vector.rs:305-313).
#pragma once
#include <cstddef>
#include <cstdint>

namespace vqb {

class CudaDevice;
struct Shape;

// up to 4096 clusters per sub-space; more than that have few rows each and are added by a scan of the codes per cluster
bool ordered_sums_applicable(size_t k);

// Sums and counts of every (sub-space, cluster), each cluster's rows added one after the other in ascending order; every
// entry of an active sub-space is overwritten.  code_bytes: width of an assignment (1 or 2).
void launch_ordered_sums(CudaDevice &dev, const Shape &sh, const float *x, const void *codes, size_t code_bytes, const uint32_t *active,
                         float *sums, uint32_t *counts, bool counts_f32);

} // namespace vqb
