// ordered_sums.cu -- cluster sums in ascending row order, as the reference's serial mean adds them (src/vector.rs:305-313).
//
// The order fixes the additions of one cluster, not the search for its rows.  So the rows are first sorted by cluster with a
// stable counting sort (two passes over the codes), and then every cluster walks its own list:
//   ordered_hist_kernel     rows per (chunk of rows, cluster)
//   ordered_lists_kernel    where each chunk's rows of a cluster start, then the row numbers themselves, ascending
//   ordered_lists_cluster_kernel  both of these, up to 65,536 rows and 1024 clusters
//   ordered_sums_kernel     one lane per (cluster, dimension) adds the cluster's rows in list order
//   ordered_sums_long_kernel the same with eight warps per list, for wide rows
// The work is O(n) per sub-space.  Walking all n codes once per (cluster, dimension), as this did before, cost 0.44 ms per pass
// at 10,000 x 128, m 16, k 256 and 1.5 ms at 33,506 x 128, k 62; three launches of this file take ~0.02 ms and ~0.05 ms.
#include <cooperative_groups.h>

#include <algorithm>

#include "cuda_device.hpp"
#include "kernels_common.cuh"
#include "ordered_sums.cuh"
#include "row_walk.cuh"

namespace vqb {

namespace cg = cooperative_groups;

namespace {

// (what the kernel before wrote is read with ordinary loads, also in row_walk.cuh: kernels_common.cuh, after_previous_kernel)
constexpr int OL_WARPS = 8, OL_THREADS = 32 * OL_WARPS;
constexpr unsigned OL_STEP = 1024;   // a chunk is a multiple of this many rows
constexpr unsigned OL_CHUNKS = 64;   // at most about this many chunks: every list CTA reads the counts of all of them
constexpr int OL_MAX_K = 4096;       // counters of eight warps in shared memory: 128 KiB
constexpr int OS_WARPS = 2; // 16 KiB of ring each

template <typename CodeT>
__global__ void __launch_bounds__(OL_THREADS) ordered_hist_kernel(const CodeT *codes, unsigned n, unsigned chunk, int m, int k,
                                                                  const uint32_t *active, uint32_t *__restrict__ hist)
{
    extern __shared__ uint32_t s_cnt[]; // [k]
    const int s = blockIdx.y;
    after_previous_kernel();
    next_kernel_may_start();
    if (active && active[s] == 0) return;
    for (int j = threadIdx.x; j < k; j += OL_THREADS) s_cnt[j] = 0u;
    __syncthreads();
    const unsigned r0 = blockIdx.x * chunk, r1 = min(n, r0 + chunk);
    for (unsigned r = r0 + threadIdx.x; r < r1; r += OL_THREADS) atomicAdd(s_cnt + (unsigned)codes[(size_t)r * m + s], 1u);
    __syncthreads();
    uint32_t *h = hist + ((size_t)s * gridDim.x + blockIdx.x) * k;
    for (int j = threadIdx.x; j < k; j += OL_THREADS) h[j] = s_cnt[j];
}

// One CTA per (chunk, sub-space).  A warp owns a contiguous eighth of the chunk, so ranking by (earlier chunks, earlier warps of
// the CTA, earlier steps of the warp, lower lanes) is ranking by row number.
template <typename CodeT>
__global__ void __launch_bounds__(OL_THREADS) ordered_lists_kernel(const CodeT *codes, unsigned n, unsigned chunk, int m, int k,
                                                                   const uint32_t *active, const uint32_t *hist,
                                                                   uint32_t *__restrict__ start, uint32_t *__restrict__ list)
{
    extern __shared__ uint32_t s_at[]; // [OL_WARPS][k]: counts, then the next free place of each list
    __shared__ uint32_t s_part[OL_WARPS];
    const int s = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    after_previous_kernel();
    next_kernel_may_start();
    if (active && active[s] == 0) return;
    const unsigned nchunks = gridDim.x, c = blockIdx.x;
    const unsigned per = chunk / OL_WARPS, w0 = c * chunk + warp * per, w1 = min(n, w0 + per);
    for (int t = threadIdx.x; t < OL_WARPS * k; t += OL_THREADS) s_at[t] = 0u;
    __syncthreads();
    uint32_t *mine = s_at + warp * k;
    for (unsigned r = w0 + lane; r < w1; r += 32) atomicAdd(mine + (unsigned)codes[(size_t)r * m + s], 1u);
    __syncthreads();
    // thread t: clusters t * jt .. t * jt + jt - 1
    const int jt = (k + OL_THREADS - 1) / OL_THREADS, j0 = threadIdx.x * jt;
    uint32_t total = 0;
    for (int j = j0; j < min(k, j0 + jt); ++j) {
        const uint32_t *h = hist + (size_t)s * nchunks * k + j;
#pragma unroll 8
        for (unsigned q = 0; q < nchunks; ++q) total += h[(size_t)q * k];
    }
    uint32_t incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_part[warp] = incl;
    __syncthreads();
    uint32_t at = incl - total;
    for (int w = 0; w < warp; ++w) at += s_part[w];
    for (int j = j0; j < min(k, j0 + jt); ++j) {
        if (c == 0) start[(size_t)s * (k + 1) + j] = at;
        const uint32_t *h = hist + (size_t)s * nchunks * k + j;
        uint32_t before = 0, all = 0;
#pragma unroll 8
        for (unsigned q = 0; q < nchunks; ++q) {
            const uint32_t v = h[(size_t)q * k];
            all += v;
            before += q < c ? v : 0u;
        }
        uint32_t place = at + before;
        for (int w = 0; w < OL_WARPS; ++w) {
            const uint32_t cnt = s_at[w * k + j];
            s_at[w * k + j] = place;
            place += cnt;
        }
        at += all;
    }
    if (c == 0 && threadIdx.x == 0) start[(size_t)s * (k + 1) + k] = n;
    __syncthreads();
    uint32_t *out = list + (size_t)s * n;
    for (unsigned r = w0 + lane; r < ((w1 + 31) & ~31u); r += 32) { // per and w0 are multiples of 32: whole warps
        const bool in = r < w1;
        const uint32_t code = in ? (uint32_t)codes[(size_t)r * m + s] : 0xFFFFFFFFu;
        const unsigned same = __match_any_sync(0xffffffffu, code);
        const int rank = __popc(same & ((1u << lane) - 1u));
        uint32_t place = 0;
        if (in) place = mine[code] + rank;
        __syncwarp();
        if (in) {
            out[place] = r;
            if (rank == 0) mine[code] += __popc(same);
        }
        __syncwarp();
    }
}

// Both steps in one launch: a cluster of CTAs per sub-space, which exchange their counts through distributed shared memory.
constexpr int OC_CTAS = 8, OC_WARPS = 16, OC_THREADS = 32 * OC_WARPS, OC_MAX_K = 1024; // counters of sixteen warps: 64 KiB
constexpr unsigned OC_STEPS = 16, OC_MAX_ROWS = OC_CTAS * OC_WARPS * 32 * OC_STEPS; // a lane keeps its rows' codes in registers: 65,536 rows

template <typename CodeT>
__global__ void __launch_bounds__(OC_THREADS) ordered_lists_cluster_kernel(const CodeT *codes, unsigned n, unsigned per, int m, int k, const uint32_t *active,
                                                                           uint32_t *__restrict__ start, uint32_t *__restrict__ list)
{
    extern __shared__ uint32_t oc_smem[]; // [OC_WARPS][k]: counts, then the next free place of each list; [k]: counts of this CTA
    __shared__ uint32_t s_part[OC_WARPS];
    cg::cluster_group cl = cg::this_cluster();
    const int s = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint32_t *s_at = oc_smem, *s_own = oc_smem + OC_WARPS * k;
    for (int t = threadIdx.x; t < OC_WARPS * k; t += OC_THREADS) s_at[t] = 0u;
    after_previous_kernel();
    next_kernel_may_start();
    if (active && active[s] == 0) return; // the whole cluster
    const unsigned c = cl.block_rank(), w0 = (c * OC_WARPS + warp) * per, w1 = min(n, w0 + per); // a warp owns `per` rows in a row, a multiple of 32
    __syncthreads();
    uint32_t *mine = s_at + warp * k;
    uint32_t code[OC_STEPS]; // all on their way at once
#pragma unroll
    for (unsigned i = 0; i < OC_STEPS; ++i) {
        const unsigned r = w0 + 32 * i + lane;
        code[i] = 32 * i < per && r < w1 ? (uint32_t)codes[(size_t)r * m + s] : 0xFFFFFFFFu;
    }
#pragma unroll
    for (unsigned i = 0; i < OC_STEPS; ++i)
        if (32 * i < per && code[i] != 0xFFFFFFFFu) atomicAdd(mine + code[i], 1u);
    __syncthreads();
    for (int j = threadIdx.x; j < k; j += OC_THREADS) {
        uint32_t total = 0;
#pragma unroll
        for (int w = 0; w < OC_WARPS; ++w) total += s_at[w * k + j];
        s_own[j] = total;
    }
    cl.sync();
    // thread t: clusters t jt .. t jt + jt - 1
    const int jt = (k + OC_THREADS - 1) / OC_THREADS, j0 = threadIdx.x * jt;
    constexpr int JT = OC_MAX_K / OC_THREADS;
    uint32_t all[JT], before[JT], total = 0;
#pragma unroll
    for (int i = 0; i < JT; ++i) {
        all[i] = before[i] = 0u;
        if (i >= jt || j0 + i >= k) continue;
#pragma unroll
        for (unsigned q = 0; q < OC_CTAS; ++q) {
            const uint32_t v = *cl.map_shared_rank(s_own + j0 + i, q);
            all[i] += v;
            before[i] += q < c ? v : 0u;
        }
        total += all[i];
    }
    uint32_t incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_part[warp] = incl;
    cl.barrier_arrive(); // (everybody has read the others' counts once this completes: before leaving)
    __syncthreads();
    uint32_t at = incl - total;
    for (int w = 0; w < warp; ++w) at += s_part[w];
#pragma unroll
    for (int i = 0; i < JT; ++i) {
        const int j = j0 + i;
        if (i >= jt || j >= k) continue;
        if (c == 0) start[(size_t)s * (k + 1) + j] = at;
        uint32_t place = at + before[i];
#pragma unroll
        for (int w = 0; w < OC_WARPS; ++w) {
            const uint32_t cnt = s_at[w * k + j];
            s_at[w * k + j] = place;
            place += cnt;
        }
        at += all[i];
    }
    if (c == 0 && threadIdx.x == 0) start[(size_t)s * (k + 1) + k] = n;
    __syncthreads();
    uint32_t *out = list + (size_t)s * n;
#pragma unroll
    for (unsigned i = 0; i < OC_STEPS; ++i) {
        if (32 * i >= per) break;
        const bool in = code[i] != 0xFFFFFFFFu;
        const unsigned same = __match_any_sync(0xffffffffu, code[i]);
        const int rank = __popc(same & ((1u << lane) - 1u));
        uint32_t place = 0;
        if (in) place = mine[code[i]] + rank;
        __syncwarp();
        if (in) {
            out[place] = w0 + 32 * i + lane;
            if (rank == 0) mine[code[i]] += __popc(same);
        }
        __syncwarp();
    }
    cl.barrier_wait();
}

// A warp takes 32 / W clusters side by side, W lanes each (W: the power of two that covers the width, at most 32; wider rows
// are cut into pieces of 32) and walks their lists (row_walk.cuh).
template <int W, bool VEC>
__global__ void __launch_bounds__(32 * OS_WARPS) ordered_sums_kernel(const float *__restrict__ x, unsigned n, unsigned long long ld, int m, int k, int sd,
                                                                     const uint32_t *active, const uint32_t *start,
                                                                     const uint32_t *list, float *sums, uint32_t *counts, int counts_f32)
{
    __shared__ __align__(16) WalkRing ring[OS_WARPS];
    const int s = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    after_previous_kernel();
    next_kernel_may_start();
    if (active && active[s] == 0) return;
    const int pieces = (sd + 31) / 32; // 1 unless W == 32
    const int unit = blockIdx.x * OS_WARPS + warp;
    const int j = (unit / pieces) * (32 / W) + lane / W, d0 = (unit % pieces) * 32, d = d0 + lane % W;
    uint32_t b = 0, len = 0;
    if (j < k) {
        b = start[(size_t)s * (k + 1) + j];
        len = start[(size_t)s * (k + 1) + j + 1] - b;
    }
    float acc = 0.0f;
    walk_rows<W, VEC>(ring[warp], x + (size_t)s * sd + d0, ld, list + (size_t)s * n + b, len, sd - d0, [&](float v) { acc = __fadd_rn(acc, v); });
    if (j < k && d < sd) {
        sums[((size_t)s * k + j) * sd + d] = acc;
        if (d == 0) counts[(size_t)s * k + j] = counts_f32 ? __float_as_uint((float)len) : len;
    }
}

// Few clusters of wide rows, whose lists are long (in the later stages of a residual fit most rows are closest to one centroid): a CTA per
// (cluster, 32 dimensions) (stream_rows).
template <bool VEC>
__global__ void __launch_bounds__(STREAM_THREADS) ordered_sums_long_kernel(const float *__restrict__ x, unsigned n, unsigned long long ld, int m, int k, int sd,
                                                                          const uint32_t *active, const uint32_t *start,
                                                                          const uint32_t *list, float *sums, uint32_t *counts, int counts_f32)
{
    extern __shared__ __align__(16) float ol_ring[];
    const int s = blockIdx.y, lane = threadIdx.x & 31;
    after_previous_kernel();
    next_kernel_may_start();
    if (active && active[s] == 0) return;
    const int pieces = (sd + 31) / 32, j = blockIdx.x / pieces, d0 = blockIdx.x % pieces * 32, cols = min(32, sd - d0);
    const uint32_t b = start[(size_t)s * (k + 1) + j], len = start[(size_t)s * (k + 1) + j + 1] - b;
    float acc = 0.0f;
    stream_rows<VEC>(ol_ring, x + (size_t)s * sd + d0, ld, list + (size_t)s * n + b, len, cols, [&](float v) { acc = __fadd_rn(acc, v); }, [](uint32_t) {});
    if (threadIdx.x >= 32 * STREAM_PRODUCERS && lane < cols) {
        sums[((size_t)s * k + j) * sd + d0 + lane] = acc;
        if (d0 + lane == 0) counts[(size_t)s * k + j] = counts_f32 ? __float_as_uint((float)len) : len;
    }
}

} // namespace

bool ordered_sums_applicable(size_t k) { return k <= (size_t)OL_MAX_K; }

template <typename CodeT>
static void launch_t(CudaDevice &dev, const Shape &sh, const float *x, const CodeT *codes, const uint32_t *active, float *sums, uint32_t *counts,
                     int counts_f32)
{
    const unsigned n = (unsigned)sh.n_local;
    const int m = (int)sh.m, k = (int)sh.k, sd = (int)sh.sd;
    const unsigned chunk = std::max(1u, ((n + OL_CHUNKS - 1) / OL_CHUNKS + OL_STEP - 1) / OL_STEP) * OL_STEP;
    const unsigned chunks = std::max(1u, (n + chunk - 1) / chunk);
    const size_t hist_words = (size_t)m * chunks * k, start_words = (size_t)m * (k + 1), list_words = (size_t)m * n;
    uint32_t *work = static_cast<uint32_t *>(dev.alloc((hist_words + start_words + list_words) * sizeof(uint32_t)));
    uint32_t *hist = work, *start = hist + hist_words, *list = start + start_words;
    // One launch instead of two, us a fit of 10 iterations: 60,000 x 128, m 16, k 256 1050 -> 950; 10,000 626 -> 608; 30,000, m 32, k 64 887 -> 864;
    // residual 33,506 x 128, k 62, 3 stages 2260 -> 2180, 5,000 x 27, k 60 1473 -> 1402 (2,500 x 128, k 256 495 -> 505).
    if (k <= OC_MAX_K && n <= OC_MAX_ROWS) {
        KernelScope ks(dev, "ordered_lists");
        auto kernel = ordered_lists_cluster_kernel<CodeT>;
        const size_t smem = sizeof(uint32_t) * (OC_WARPS + 1) * k;
        allow_shared_memory(dev, kernel);
        const unsigned per = ((n + OC_CTAS * OC_WARPS - 1) / (OC_CTAS * OC_WARPS) + 31) / 32 * 32;
        launch_following_clusters(kernel, dim3(OC_CTAS, m), OC_THREADS, smem, OC_CTAS, dev.stream(), codes, n, per, m, k, active, start, list);
        dev.count_launch();
    } else {
        KernelScope ks(dev, "ordered_lists");
        const size_t smem = sizeof(uint32_t) * k;
        launch_following(ordered_hist_kernel<CodeT>, dim3(chunks, m), OL_THREADS, smem, dev.stream(), codes, n, chunk, m, k, active, hist);
        dev.count_launch();
        auto kernel = ordered_lists_kernel<CodeT>;
        allow_shared_memory(dev, kernel);
        launch_following(kernel, dim3(chunks, m), OL_THREADS, OL_WARPS * smem, dev.stream(), codes, n, chunk, m, k, active, hist, start, list);
        dev.count_launch();
    }
    const bool vec = sd % 4 == 0 && sh.ld % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0; // whole 16-byte pieces
    const size_t long_units = (size_t)k * ((sd + 31) / 32);
    // Both kernels (us): 20,423 rows, k 16, 61-wide 308 walked / 85 here, k 62 34 / 15; 60,000 rows, k 16, 128-wide 437 / 153, k 100 30 / 16, k 256 (1024
    // CTAs) 20 / 17; 2000 rows, k 100, 128-wide 10.1 / 8.7; but 1024 CTAs with lists of 23 rows 9.5 / 10.6, of 79 rows 12.1 / 12.7.
    if (sd > 16 && (long_units * m <= (size_t)dev.sm_count() * 4 || n / k >= 150)) {
        KernelScope ks(dev, "ordered_sums");
        auto kernel = vec ? ordered_sums_long_kernel<true> : ordered_sums_long_kernel<false>;
        VQB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STREAM_SMEM));
        launch_following(kernel, dim3((unsigned)long_units, m), STREAM_THREADS, STREAM_SMEM, dev.stream(), x, n, sh.ld, m, k, sd, active, start, list, sums, counts,
                         counts_f32);
        dev.count_launch();
    } else {
        KernelScope ks(dev, "ordered_sums");
        const int w = sd <= 4 ? 4 : sd <= 8 ? 8 : sd <= 16 ? 16 : 32;
        const size_t units = ((size_t)k + 32 / w - 1) / (32 / w) * ((sd + 31) / 32);
        const dim3 grid((unsigned)((units + OS_WARPS - 1) / OS_WARPS), m);
        // Up to a block per SM: launched while the kernel before them runs, the blocks would gather on the SMs that are free first and share
        // one port for their scattered 16-byte copies.  They ask for half of an SM's shared memory, so that no two share one.  Fits of 5
        // iterations, launched after the kernel before / overlapping it / like this: 60,000 rows, 16 sub-spaces of 4, k 16 1151 / 1545 / 962 us;
        // 30,000 rows, 32 of 4, k 16 808 / 984 / 728; 10,000 rows, 8 of 4, k 16 371 / 321 / 321.  (Two to six blocks spread the same
        // way: 64 of 4, k 64 8 % faster, 32 of 8, 2500 rows, k 256 3 % slower.)
        const size_t rings = sizeof(WalkRing) * OS_WARPS;
        const size_t spread = (size_t)grid.x * grid.y <= (size_t)dev.sm_count() && dev.smem_limit() / 2 > rings ? dev.smem_limit() / 2 - rings : 0;
        auto go = [&](auto kernel) {
            if (spread) allow_shared_memory(dev, kernel);
            launch_following(kernel, grid, 32 * OS_WARPS, spread, dev.stream(), x, n, sh.ld, m, k, sd, active, start, list, sums, counts, counts_f32);
        };
        if (w == 4) go(vec ? ordered_sums_kernel<4, true> : ordered_sums_kernel<4, false>);
        else if (w == 8) go(vec ? ordered_sums_kernel<8, true> : ordered_sums_kernel<8, false>);
        else if (w == 16) go(vec ? ordered_sums_kernel<16, true> : ordered_sums_kernel<16, false>);
        else go(vec ? ordered_sums_kernel<32, true> : ordered_sums_kernel<32, false>);
        dev.count_launch();
    }
    dev.release(work);
}

void launch_ordered_sums(CudaDevice &dev, const Shape &sh, const float *x, const void *codes, size_t code_bytes, const uint32_t *active, float *sums,
                         uint32_t *counts, bool counts_f32)
{
    const int cf = counts_f32 ? 1 : 0;
    if (code_bytes == 1) launch_t(dev, sh, x, static_cast<const uint8_t *>(codes), active, sums, counts, cf);
    else launch_t(dev, sh, x, static_cast<const uint16_t *>(codes), active, sums, counts, cf);
}

} // namespace vqb
