// direct.cuh -- encoding few rows in one launch (direct.cu).
#pragma once
#include <cstddef>
#include <cstdint>

#include "assign_generic.cuh"
#include "assign_reg.cuh"

namespace vqb {

class CudaDevice;

// Whether the one-launch kernel is the better one for an encode of this size; tensor: the alternative is the tensor-core path.
bool direct_encode_applicable(const AssignParams &p, bool tensor);
void launch_direct_encode(CudaDevice &dev, const AssignParams &p, int metric);

// The same for the residual encoder: all stages of a row in one launch.  g.m == 1, g.centroids [stages][k][sd].
bool direct_rvq_applicable(const GenericParams &g, size_t smem_limit);
void launch_direct_rvq(CudaDevice &dev, const GenericParams &g, int metric);

} // namespace vqb
