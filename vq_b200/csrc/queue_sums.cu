// queue_sums.cu -- cluster sums and counts of narrow sub-spaces (src/utils.rs:83-92 + src/vector.rs:297-314, no fixed order).
//
// f32 atomics in shared memory are loops of compare-and-swap, one per element: a row slice of 8 dimensions that changes its
// cluster took 16 of them.  Here every cluster of a CTA belongs to one team of lanes (a lane per 16 bytes), so nothing needs an
// atomic but the place in a queue: in step one a thread looks at the codes of its rows and appends each (row, cluster) to the
// queue of the cluster's team; in step two the teams fetch the queued slices from memory, four at a time, and add them to
// their clusters' sums in shared memory with ordinary 128-bit loads and stores.  A full queue is no error, its overflow goes
// straight to global memory.
//
// Clusters are numbered bin = code * G + sub-space; team = bin modulo the number of teams, so the teams of a quarter-warp always
// touch different banks.
//
// Measured, moves of k-means iterations, mean of nine: 1M x 128 in 16 sub-spaces, k 256: 117 -> 77 us; 500,000 x 64, 16: 98 -> 39;
// 400,000 x 256, 8: 179 -> 57.  1M of 128, one sub-space: 95 -> 71; 400,000 of 40: 75 (all rows anew) -> 23.  All rows of the first shape: 238 -> 207 us, i.e. 2.6 TB/s of rows: the integer work of the queues
// (2.2 instructions a cycle) and the trip to memory in front of every four additions share the time.
#include <algorithm>

#include "cuda_device.hpp"
#include "kernels_common.cuh"
#include "queue_sums.cuh"

namespace vqb {

namespace {

constexpr int QS_ROWS = 2048, QS_BATCH = 4;
// two CTAs of 512 threads per SM; wide rows leave room for the sums of one
__host__ __device__ constexpr int qs_threads(int le) { return le == 32 ? 1024 : 512; }
// a queue entry: row within the piece (11 bits), bin / teams (4 bits), sign
constexpr int QS_ROW_BITS = 11, QS_MAX_BINS_PER_TEAM = 16;
static_assert(QS_ROWS / 512 * 8 <= 32, "a bit per entry of a thread");
static_assert(QS_ROWS == 1 << QS_ROW_BITS, "a row of a piece has to fit its bits");

struct QsParams {
    const float *x;
    unsigned long long n, ld, rows_per_cta;
    int m, k, sd, cap;
    uint8_t *prev;
    const uint8_t *codes;
    const uint32_t *active;
    float *sums;
    uint32_t *counts;
    int counts_f32;
};

__device__ __forceinline__ void qs_count(const QsParams &P, size_t at, int c)
{
    if (P.counts_f32) atomicAdd(reinterpret_cast<float *>(P.counts) + at, (float)c);
    else atomicAdd(P.counts + at, (uint32_t)c); // modulo 2^32: the total is the true count
}

// LE: lanes per team (a power of two, 4 * LE >= sd); G: sub-spaces per CTA; MOVED: codes_prev is given
template <int LE, int G, bool MOVED>
__global__ void __launch_bounds__(qs_threads(LE), 1024 / qs_threads(LE)) queue_sums_kernel(const QsParams P)
{
    constexpr int QS_THREADS = qs_threads(LE), QS_PER = QS_ROWS / QS_THREADS;
    constexpr int TEAMS = QS_THREADS / LE;
    extern __shared__ __align__(16) unsigned char qs_smem[];
    const int bins = P.k * G, g0 = blockIdx.y * G, gc = min(G, P.m - g0);
    float *ssum = reinterpret_cast<float *>(qs_smem);               // [bins][sd]
    int *scnt = reinterpret_cast<int *>(ssum + (size_t)bins * P.sd); // [bins]
    uint32_t *fill = reinterpret_cast<uint32_t *>(scnt + bins);      // [TEAMS]
    uint16_t *queue = reinterpret_cast<uint16_t *>(fill + TEAMS);    // [cap][TEAMS]
    for (int t = threadIdx.x; t < bins * P.sd; t += QS_THREADS) ssum[t] = 0.0f;
    for (int t = threadIdx.x; t < bins; t += QS_THREADS) scnt[t] = 0;
    if (threadIdx.x < TEAMS) fill[threadIdx.x] = 0;
    after_previous_kernel();
    next_kernel_may_start();
    uint32_t live = 0; // byte mask of the sub-spaces that take part
    for (int sl = 0; sl < gc; ++sl)
        if (!P.active || P.active[g0 + sl] != 0) live |= 0xFFu << (8 * sl);
    __syncthreads();

    const unsigned long long first = blockIdx.x * P.rows_per_cta;
    const unsigned rows = first < P.n ? (unsigned)min(P.rows_per_cta, P.n - first) : 0u;
    const unsigned pieces = (rows + QS_ROWS - 1) / QS_ROWS, piece = pieces ? (rows + pieces - 1) / pieces : 0u;
    const bool words = G == 4 && P.m % 4 == 0 && ((reinterpret_cast<uintptr_t>(P.codes) | reinterpret_cast<uintptr_t>(P.prev)) & 3u) == 0;
    const int team = threadIdx.x / LE, part = threadIdx.x % LE;
    const bool has_part = 4 * part < P.sd;
    // G divides the number of teams, so a team's clusters are all of one sub-space
    const uint32_t ld = (uint32_t)P.ld, stride = (uint32_t)(TEAMS * P.sd);
    const size_t xcol = (size_t)(g0 + team % G) * P.sd + 4 * part;
    float *mine = ssum + team * P.sd + 4 * part;

    auto load = [&](const uint8_t *codes, unsigned long long row) {
        const uint8_t *p = codes + row * P.m + g0;
        if (words) return *reinterpret_cast<const uint32_t *>(p);
        uint32_t w = 0;
        for (int sl = 0; sl < gc; ++sl) w |= (uint32_t)p[sl] << (8 * sl);
        return w;
    };
    uint32_t now[QS_PER], was[QS_PER];
    auto load_piece = [&](unsigned i) {
#pragma unroll
        for (int r = 0; r < QS_PER; ++r) {
            const unsigned in = threadIdx.x + r * QS_THREADS;
            now[r] = was[r] = 0;
            if (in < piece && i * piece + in < rows) {
                const unsigned long long row = first + i * piece + in;
                now[r] = load(P.codes, row);
                if (MOVED) was[r] = load(P.prev, row);
            }
        }
    };
    auto ahead = [&](unsigned long long row, int sl, int d = 0) { // towards L2, from where the teams fetch it
        asm volatile("prefetch.global.L2 [%0];" ::"l"(P.x + row * P.ld + (size_t)(g0 + sl) * P.sd + d));
    };
    // appends row `in` of the piece to the queue of its cluster; bit `id` of `over` is set if that is full
    uint32_t over = 0;
    auto append = [&](unsigned in, int sl, uint32_t code, uint32_t minus, int id) {
        const uint32_t bin = code * G + sl, to = bin % TEAMS;
        atomicAdd(scnt + bin, minus ? -1 : 1);
        const uint32_t at = atomicAdd(fill + to, 1u);
        if (at < (uint32_t)P.cap) queue[at * TEAMS + to] = (uint16_t)(in | (bin / TEAMS) << QS_ROW_BITS | minus << 15);
        else over |= 1u << id;
    };
    if (pieces) load_piece(0);
    for (unsigned i = 0; i < pieces; ++i) {
        const unsigned long long row0 = first + i * piece;
#pragma unroll
        for (int r = 0; r < QS_PER; ++r) {
            const unsigned in = threadIdx.x + r * QS_THREADS;
            if (MOVED) {
                uint32_t diff = (was[r] ^ now[r]) & live;
                if (diff == 0) continue; // rows that are not there, too
                uint8_t *prev = P.prev + (row0 + in) * P.m + g0;
                if (words) *reinterpret_cast<uint32_t *>(prev) = (was[r] & ~live) | (now[r] & live);
                while (diff) { // unlike the unrolled form, a warp's steps are the moves of its busiest row
                    const int sl = (__ffs((int)diff) - 1) >> 3;
                    diff &= ~(0xFFu << (8 * sl));
                    if (!words) prev[sl] = (uint8_t)(now[r] >> (8 * sl));
                    ahead(row0 + in, sl);
                    append(in, sl, (now[r] >> (8 * sl)) & 0xFFu, 0u, (r * 4 + sl) * 2);
                    append(in, sl, (was[r] >> (8 * sl)) & 0xFFu, 1u, (r * 4 + sl) * 2 + 1);
                }
            } else if (in < piece && i * piece + in < rows) {
                for (int d = 0; d < gc * P.sd; d += 32) ahead(row0 + in, 0, d);
#pragma unroll
                for (int sl = 0; sl < G; ++sl)
                    if (live >> (8 * sl) & 1u) append(in, sl, (now[r] >> (8 * sl)) & 0xFFu, 0u, (r * 4 + sl) * 2);
            }
        }
        for (; over; over &= over - 1) { // what found its queue full goes straight to global memory (its count is taken)
            const int id = __ffs((int)over) - 1, sl = id >> 1 & 3;
            uint32_t word = 0;
#pragma unroll
            for (int r = 0; r < QS_PER; ++r)
                if (id >> 3 == r) word = id & 1 ? was[r] : now[r];
            const float *xp = P.x + (row0 + threadIdx.x + (id >> 3) * QS_THREADS) * P.ld + (size_t)(g0 + sl) * P.sd;
            float *to = P.sums + ((size_t)(g0 + sl) * P.k + ((word >> (8 * sl)) & 0xFFu)) * P.sd;
            const float sign = id & 1 ? -1.0f : 1.0f;
            for (int d = 0; d < P.sd; d += 4) {
                const float4 v = __ldg(reinterpret_cast<const float4 *>(xp + d));
                atomicAdd(reinterpret_cast<float4 *>(to + d), make_float4(sign * v.x, sign * v.y, sign * v.z, sign * v.w));
            }
        }
        __syncthreads();
        if (i + 1 < pieces) load_piece(i + 1);
        const uint32_t count = min(fill[team], (uint32_t)P.cap);
        __syncwarp(); // the team's lanes have read its count
        if (part == 0) fill[team] = 0;
        const float *xp = P.x + row0 * P.ld + xcol;
        for (uint32_t e0 = 0; e0 < count; e0 += QS_BATCH) {
            uint32_t e[QS_BATCH];
            float4 v[QS_BATCH];
#pragma unroll
            for (int b = 0; b < QS_BATCH; ++b)
                if (e0 + b < count) {
                    e[b] = queue[(e0 + b) * TEAMS + team];
                    if (has_part) v[b] = __ldg(reinterpret_cast<const float4 *>(xp + (unsigned long long)(e[b] & (QS_ROWS - 1)) * ld));
                }
#pragma unroll
            for (int b = 0; b < QS_BATCH; ++b)
                if (e0 + b < count && has_part) {
                    float4 *s = reinterpret_cast<float4 *>(mine + (e[b] >> QS_ROW_BITS & (QS_MAX_BINS_PER_TEAM - 1)) * stride);
                    const float sign = MOVED && e[b] >> 15 ? -1.0f : 1.0f;
                    float4 t = *s;
                    t.x = fmaf(sign, v[b].x, t.x), t.y = fmaf(sign, v[b].y, t.y), t.z = fmaf(sign, v[b].z, t.z), t.w = fmaf(sign, v[b].w, t.w);
                    *s = t;
                }
        }
        __syncthreads(); // the queues are empty
    }
    const int quarter = P.sd / 4;
    for (int t = threadIdx.x; t < bins * quarter; t += QS_THREADS) {
        const int bin = t / quarter, d = t % quarter * 4, sl = bin % G, j = bin / G;
        const float4 v = *reinterpret_cast<const float4 *>(ssum + (size_t)bin * P.sd + d);
        if (sl < gc && (v.x != 0.0f || v.y != 0.0f || v.z != 0.0f || v.w != 0.0f))
            atomicAdd(reinterpret_cast<float4 *>(P.sums + ((size_t)(g0 + sl) * P.k + j) * P.sd + d), v);
    }
    for (int t = threadIdx.x; t < bins; t += QS_THREADS)
        if (scnt[t] != 0) qs_count(P, (size_t)(g0 + t % G) * P.k + t / G, scnt[t]);
}

struct Plan {
    int le, g, cap;
    size_t smem;
};

// Four sub-spaces per CTA (their codes are one word, their slices of a row adjacent), fewer where their sums would leave room for
// one CTA per SM only.  A queue takes one and a half times the average of a pass over all rows.
Plan plan(size_t m, size_t k, size_t sd, size_t budget)
{
    Plan p = {1, 4, 0, 0};
    while (4 * (size_t)p.le < sd) p.le *= 2;
    if (p.le > 8) p.le = 32, p.g = 1;
    const int teams = qs_threads(p.le) / p.le;
    while (p.g > 1 && (size_t)p.g / 2 >= m) p.g /= 2;
    for (;; p.g /= 2) {
        p.cap = QS_ROWS * p.g / teams * 3 / 2 + 32;
        p.smem = k * p.g * (sd + 1) * 4 + (size_t)teams * (4 + 2 * p.cap);
        if (p.g == 1 || (p.smem <= budget / 2 && k * p.g <= (size_t)teams * QS_MAX_BINS_PER_TEAM)) return p;
    }
}

template <int LE, int G> void launch(CudaDevice &dev, const QsParams &q, dim3 grid, size_t smem)
{
    auto kernel = q.prev ? queue_sums_kernel<LE, G, true> : queue_sums_kernel<LE, G, false>;
    allow_shared_memory(dev, kernel);
    launch_following(kernel, grid, qs_threads(LE), smem, dev.stream(), q);
    dev.count_launch();
}

template <int LE> void launch(CudaDevice &dev, const QsParams &q, int g, dim3 grid, size_t smem)
{
    if (g == 4) launch<LE, 4>(dev, q, grid, smem);
    else if (g == 2) launch<LE, 2>(dev, q, grid, smem);
    else launch<LE, 1>(dev, q, grid, smem);
}

} // namespace

bool queue_sums_applicable(CudaDevice &dev, const Shape &sh, const float *x, const float *sums, size_t code_bytes, bool moved)
{
    // all rows of wide sub-spaces: accum_owner_kernel streams them without queues (1M x 128, k 256: 213 us against 300 and more)
    if (code_bytes != 1 || sh.sd < 4 || sh.sd > (moved ? 128 : 32) || sh.sd % 4 || sh.ld % 4 || sh.m > 65535u || sh.ld >> 32 || sh.n_local >= (1ull << 40)) return false;
    return ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(sums)) & 15u) == 0 && plan(sh.m, sh.k, sh.sd, dev.smem_limit() - 4096).smem <= dev.smem_limit() - 1024;
}

void launch_queue_sums(CudaDevice &dev, const Shape &sh, const float *x, uint8_t *codes_prev, const uint8_t *codes, const uint32_t *active, float *sums,
                       uint32_t *counts, bool counts_f32)
{
    if (sh.n_local == 0) return;
    const Plan p = plan(sh.m, sh.k, sh.sd, dev.smem_limit() - 4096);
    const unsigned ny = (unsigned)((sh.m + p.g - 1) / p.g);
    const size_t per_sm = p.le < 32 && p.smem <= (dev.smem_limit() - 4096) / 2 ? 2 : 1;
    size_t gx = std::max<size_t>(1, (size_t)dev.sm_count() * per_sm / ny);
    gx = std::min<size_t>(gx, (sh.n_local + 511) / 512);
    gx = std::max<size_t>(gx, sh.n_local >> 30); // row numbers within a CTA are 32 bits wide
    QsParams q = {x, sh.n_local, sh.ld, (sh.n_local + gx - 1) / gx, (int)sh.m, (int)sh.k, (int)sh.sd, p.cap, codes_prev, codes, active, sums, counts, counts_f32 ? 1 : 0};
    KernelScope ks(dev, codes_prev ? "accumulate_moved" : "accumulate_fast");
    const dim3 grid((unsigned)gx, ny);
    if (p.le == 1) launch<1>(dev, q, p.g, grid, p.smem);
    else if (p.le == 2) launch<2>(dev, q, p.g, grid, p.smem);
    else if (p.le == 4) launch<4>(dev, q, p.g, grid, p.smem);
    else if (p.le == 8) launch<8>(dev, q, p.g, grid, p.smem);
    else launch<32, 1>(dev, q, grid, p.smem);
}

} // namespace vqb
