// row_walk.cuh -- a warp walks lists of rows in order, for sums whose order is part of the result.
//
// W lanes take one list each (32 / W lists side by side; W = 4, 8, 16 or 32), lane = dimension, use(v) is called once per row of the
// list, in order.  What is done with the values is one dependent chain of a few cycles a row, so all of the way to memory has to
// lie ahead of it: 96 rows travel through a shared-memory ring (cp.async) and the row numbers are read another 32 rows
// earlier, 32 at a time.  (Numbers read one batch of eight ahead cost a round trip to L2 per batch: 97 cycles a row.)
// Rows of whole 16-byte pieces (VEC) travel four at a time, a piece per lane; others one at a time, an element per lane, which costs
// four times the instructions.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace vqb {

constexpr int WALK_BATCH = 8, WALK_BLOCK = 32, WALK_RING = 128; // rows: per commit group, per fetch of numbers, in the ring
typedef float WalkRing[WALK_RING][32];                          // 16 KiB per warp, 16-byte aligned

// x: column 0 of row number 0; rows: this lane's list (the same for its W lanes); count: its length; cols: the list's live
// columns, at most W of them are used (VEC: a multiple of 4, x on 16 bytes, ld a multiple of 4).  All lanes call it together.
template <int W, bool VEC, typename Use>
__device__ __forceinline__ void walk_rows(WalkRing &ring, const float *x, size_t ld, const uint32_t *rows, uint32_t count, int cols, Use &&use)
{
    constexpr int NR = WALK_BLOCK / W, AHEAD = WALK_RING / WALK_BLOCK - 1; // registers of numbers per block; blocks in flight
    constexpr int STEP = VEC ? 4 : 1, LANES = W / STEP;                   // rows per copy; lanes per row of a list
    const int lane = threadIdx.x & 31, sub = lane % W, line = sub / LANES, col = sub % LANES * STEP;
    const uint32_t most = __reduce_max_sync(0xffffffffu, count), blocks = (most + WALK_BLOCK - 1) / WALK_BLOCK;
    const bool live = col < cols;
    x += col;
    const uint32_t to = (uint32_t)__cvta_generic_to_shared(&ring[line][lane - sub + col]);
    uint32_t num[AHEAD + 1][NR];
    auto numbers = [&](uint32_t(&of)[NR], uint32_t block) {
#pragma unroll
        for (int q = 0; q < NR; ++q) {
            const uint32_t at = block * WALK_BLOCK + q * W + sub;
            of[q] = at < count ? rows[at] : 0u;
        }
    };
    auto issue = [&](const uint32_t(&of)[NR], uint32_t block, int batch) { // always closes a group: the number of pending ones stays fixed
        if (block < blocks) {
            const uint32_t slot = to + block * WALK_BLOCK % WALK_RING * 128, left = count - block * WALK_BLOCK; // (left is used where positive)
            const bool some = count > block * WALK_BLOCK && live;
#pragma unroll
            for (int i = 0; i < WALK_BATCH; i += STEP) {
                const int at = batch * WALK_BATCH + i;
                const uint32_t row = __shfl_sync(0xffffffffu, of[at / W], at % W + line, W);
                if (some && at + line < left) {
                    const float *from = x + (size_t)row * ld;
                    if (VEC)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(slot + at * 128), "l"(from) : "memory");
                    else
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(slot + at * 128), "l"(from) : "memory");
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
#pragma unroll
    for (int b = 0; b <= AHEAD; ++b) numbers(num[b], b);
#pragma unroll
    for (int b = 0; b < AHEAD; ++b)
#pragma unroll
        for (int j = 0; j < WALK_BLOCK / WALK_BATCH; ++j) issue(num[b], b, j);
#pragma unroll 1
    for (uint32_t b = 0; b < blocks; ++b) {
        numbers(num[0], b + AHEAD + 1);
#pragma unroll
        for (int j = 0; j < WALK_BLOCK / WALK_BATCH; ++j) {
            issue(num[AHEAD], b + AHEAD, j); // over rows that every lane has used before the last __syncwarp
            asm volatile("cp.async.wait_group %0;" ::"n"(AHEAD * WALK_BLOCK / WALK_BATCH) : "memory");
            __syncwarp();
            float v[WALK_BATCH];
#pragma unroll
            for (int i = 0; i < WALK_BATCH; ++i) v[i] = ring[b * WALK_BLOCK % WALK_RING + j * WALK_BATCH + i][lane];
#pragma unroll
            for (int i = 0; i < WALK_BATCH; ++i)
                if (b * WALK_BLOCK + j * WALK_BATCH + i < count) use(v[i]);
        }
#pragma unroll
        for (int q = 0; q < NR; ++q) num[AHEAD][q] = num[0][q];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
}

// The same for one long list by a whole CTA of STREAM_THREADS threads: seven warps bring the rows (stages of 128, three ahead), the eighth, lane =
// dimension, calls use(v) once per row in order, and stage_end(t) behind the last row of stage t.  7 to 8 cycles a row, where a warp that
// does everything takes 25 to 33, its instructions one after the other.
constexpr int STREAM_STAGE = 128, STREAM_SLOTS = 4, STREAM_PRODUCERS = 7, STREAM_SHARE = 20; // rows of a stage; stages in the ring; rows of a producer (7 x 20 >= 128)
constexpr int STREAM_THREADS = 32 * (STREAM_PRODUCERS + 1);
constexpr size_t STREAM_SMEM = (size_t)STREAM_SLOTS * STREAM_STAGE * 32 * sizeof(float);

// ring: STREAM_SMEM bytes, 16-byte aligned; x: column 0 of row number 0; cols: live columns, at most 32 (VEC: a multiple of 4, x on 16 bytes,
// ld a multiple of 4).  All threads call it together; afterwards the ring may be used again.
template <bool VEC, typename Use, typename StageEnd>
__device__ __forceinline__ void stream_rows(float *ring, const float *x, size_t ld, const uint32_t *rows, uint32_t len, int cols, Use &&use, StageEnd &&stage_end)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t stages = (len + STREAM_STAGE - 1) / STREAM_STAGE;
    const int first = warp * STREAM_SHARE, share = min(STREAM_SHARE, STREAM_STAGE - first); // producer warp's rows of a stage
    auto number = [&](uint32_t t) -> uint32_t {                                             // of the producer's row `lane` in stage t
        const uint32_t at = t * STREAM_STAGE + first + lane;
        return lane < share && at < len ? rows[at] : 0u;
    };
    auto issue = [&](uint32_t t, uint32_t num) { // always closes a group
        if (t < stages) {
            const int here = min(share, (int)(len - min(len, t * STREAM_STAGE + first))); // rows of this share that the list has
            float *slot = ring + ((size_t)(t % STREAM_SLOTS) * STREAM_STAGE + first) * 32;
            if (VEC) {
#pragma unroll
                for (int i = 0; i < STREAM_SHARE; i += 4) { // four rows at a time, eight lanes each
                    const int r = i + (lane >> 3), c = (lane & 7) * 4;
                    const uint32_t row = __shfl_sync(0xffffffffu, num, r);
                    if (r < here && c < cols)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(slot + r * 32 + c)), "l"(x + (size_t)row * ld + c) : "memory");
                }
            } else {
#pragma unroll
                for (int r = 0; r < STREAM_SHARE; ++r) {
                    const uint32_t row = __shfl_sync(0xffffffffu, num, r);
                    if (r < here && lane < cols)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(slot + r * 32 + lane)), "l"(x + (size_t)row * ld + lane) : "memory");
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const bool producer = warp < STREAM_PRODUCERS;
    uint32_t num = 0;
    if (producer) {
#pragma unroll
        for (uint32_t t = 0; t < STREAM_SLOTS - 1; ++t) issue(t, number(t));
        num = number(STREAM_SLOTS - 1);
    }
    for (uint32_t t = 0; t < stages; ++t) {
        if (producer) asm volatile("cp.async.wait_group %0;" ::"n"(STREAM_SLOTS - 2) : "memory"); // stage t of this warp is there
        __syncthreads();                                                                          // and of all; stage t - 1 is used up
        if (producer) {
            issue(t + STREAM_SLOTS - 1, num);
            num = number(t + STREAM_SLOTS);
        } else {
            const float *v = ring + (size_t)(t % STREAM_SLOTS) * STREAM_STAGE * 32 + lane;
            const int here = (int)min((uint32_t)STREAM_STAGE, len - t * STREAM_STAGE);
            if (here == STREAM_STAGE) {
                float cur[8], next[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) cur[i] = v[i * 32];
#pragma unroll 4
                for (int r = 8; r <= STREAM_STAGE; r += 8) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) next[i] = v[(r < STREAM_STAGE ? r + i : i) * 32];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        use(cur[i]);
                        cur[i] = next[i];
                    }
                }
            } else {
#pragma unroll 4
                for (int r = 0; r < here; ++r) use(v[r * 32]);
            }
            stage_end(t);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

} // namespace vqb
