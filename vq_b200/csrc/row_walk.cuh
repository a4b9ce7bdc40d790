// row_walk.cuh -- a warp walks lists of rows in order, for sums whose order is part of the result.
//
// W lanes take one list each (32 / W lists side by side; W = 4, 8, 16 or 32), lane = dimension, use(v) is called once per row of the
// list, in order.  What is done with the values is one dependent chain of a few cycles a row, so all of the way to memory has to
// lie ahead of it: 96 rows travel through a shared-memory ring (cp.async) and the row numbers are read another 32 rows
// earlier, 32 at a time.  (Numbers read one batch of eight ahead cost a round trip to L2 per batch: 97 cycles a row.)
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vqb {

constexpr int WALK_BATCH = 8, WALK_BLOCK = 32, WALK_RING = 128; // rows: per commit group, per fetch of numbers, in the ring
typedef float WalkRing[WALK_RING][32];                          // 16 KiB per warp

// x: the list's first row number 0 at this lane's dimension; rows: this lane's list (the same for its W lanes); count: its length;
// live: the lane has a dimension.  All lanes of the warp call it together.
template <int W, typename Use>
__device__ __forceinline__ void walk_rows(WalkRing &ring, const float *x, size_t ld, const uint32_t *rows, uint32_t count, bool live, Use &&use)
{
    constexpr int NR = WALK_BLOCK / W, AHEAD = WALK_RING / WALK_BLOCK - 1; // registers of numbers per block; blocks in flight
    const int lane = threadIdx.x & 31, sub = lane % W;
    const uint32_t most = __reduce_max_sync(0xffffffffu, count), blocks = (most + WALK_BLOCK - 1) / WALK_BLOCK;
    uint32_t now[NR], next[NR];
    auto numbers = [&](uint32_t(&to)[NR], uint32_t block) {
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            const uint32_t at = block * WALK_BLOCK + q * W + sub;
            to[q] = at < count ? __ldg(rows + at) : 0u;
        }
    };
    auto issue = [&](const uint32_t(&of)[NR], uint32_t block, int batch) { // always closes a group: the number of pending ones stays fixed
#pragma unroll
        for (int i = 0; i < WALK_BATCH; ++i) {
            const int at = batch * WALK_BATCH + i;
            const uint32_t row = __shfl_sync(0xffffffffu, of[at / W], at % W, W);
            if (block * WALK_BLOCK + at < count && live)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(&ring[(block * WALK_BLOCK + at) % WALK_RING][lane])),
                             "l"(x + (size_t)row * ld)
                             : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    numbers(now, 0);
#pragma unroll 1
    for (uint32_t b = 0; b < AHEAD; ++b) {
        numbers(next, b + 1);
#pragma unroll
        for (int j = 0; j < WALK_BLOCK / WALK_BATCH; ++j) issue(now, b, j);
#pragma unroll
        for (int q = 0; q < NR; ++q) now[q] = next[q];
    }
#pragma unroll 1
    for (uint32_t b = 0; b < blocks; ++b) {
        numbers(next, b + AHEAD + 1);
#pragma unroll
        for (int j = 0; j < WALK_BLOCK / WALK_BATCH; ++j) {
            issue(now, b + AHEAD, j);
            asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD * WALK_BLOCK / WALK_BATCH) : "memory"); // a lane reads only what it copied itself
            float v[WALK_BATCH];
#pragma unroll
            for (int i = 0; i < WALK_BATCH; ++i) v[i] = ring[(b * WALK_BLOCK + j * WALK_BATCH + i) % WALK_RING][lane];
#pragma unroll
            for (int i = 0; i < WALK_BATCH; ++i)
                if (b * WALK_BLOCK + j * WALK_BATCH + i < count) use(v[i]);
        }
#pragma unroll
        for (int q = 0; q < NR; ++q) now[q] = next[q];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

} // namespace vqb
