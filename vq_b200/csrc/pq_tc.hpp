// pq_tc.hpp -- tensor-core product-quantizer assignment (pq_tc.cu).
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda.h>

#include "iter_status.cuh"
#include "peer_exchange.cuh"
#include "pq_tc_shape.hpp"

namespace vqb {

class CudaDevice;
struct AssignParams;

// pq_tc_shape is what the kernels and the fused centroid update take: for an assignment with pq_tc_rows and 16-byte aligned row slices, for the
// Euclidean metrics or (encode) cosine
bool pq_tc_applicable(const AssignParams &p, int metric);
// whether an encode that the kernels can take is faster with them than on the CUDA cores
bool pq_tc_encode_pays(const AssignParams &p, int metric);
size_t pq_tc_scratch_floats();
// bytes of the one-byte codes that an encode of n rows of m sub-spaces goes through
size_t pq_tc_code_bytes(size_t n, size_t m);

// How TMA reads operand B from the scratch memory; made once for it.
struct PqTcMaps {
    CUtensorMap b1, b2;
};
PqTcMaps pq_tc_make_maps(const float *scratch);

// Device memory one launch works with besides its inputs and outputs.
struct PqTcBuffers {
    float *scratch = nullptr;     // pq_tc_scratch_floats() floats, zero-filled once: operand B, binary16 images, constants, statistics
    const PqTcMaps *maps = nullptr; // of scratch
    uint8_t *codes = nullptr;     // encode: pq_tc_code_bytes(n, m) bytes of working memory
    int *error_word = nullptr;    // set when a bounded wait expires
    bool prepare_operand = true;  // false: scratch already holds operand B of p.centroids (written by launch_pq_update_centroids)
    float *dbg_scores = nullptr;  // optional: n x m x 256 raw scores, or with dbg_frames (n x m x 2: sigma, K0) the fixed-point ones and no codes
    float *dbg_frames = nullptr;
};
void launch_pq_operand_b(CudaDevice &dev, const float *centroids, int m, int k, int sd, bool cosine, float *scratch);
void launch_pq_tc(CudaDevice &dev, const AssignParams &p, int metric, bool train, size_t code_bytes, const PqTcBuffers &b);
// number of (row, sub-space) pairs the tensor kernel has left to the reference's arithmetic so far (first u64 of the statistics)
size_t pq_tc_stats_offset_floats();
size_t pq_tc_consts_offset_floats(); // the sub-spaces' constants, 32 each
// centroid update + operand B of the next pass + the iteration's flags, one launch (m CTAs)
void launch_pq_update_centroids(CudaDevice &dev, int m, int k, int sd, float *sums, uint32_t *counts, uint32_t *moved, bool counts_f32,
                                const uint32_t *active, float *centroids, float *scratch, const StatusPage &sp, const PeerView &pv);

} // namespace vqb
