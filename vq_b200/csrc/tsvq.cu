// tsvq.cu -- tree-structured vector quantizer (src/tsvq.rs) built level by level on the device.
//
// The reference recurses; here all nodes of one depth are processed together and numbered breadth-first (left child before
// right).  What fixes the result bit for bit is kept: the centroid of a node is the f32 sum of its rows divided by
// `len as f32` (mean_vector, src/vector.rs:282-318), added up as the sum of the sums of consecutive 1024-row chunks -- for
// up to 1024 rows the reference's serial order, above that one admissible order where the reference's own parallel
// reduction is unspecified, and one whose chunks can be added side by side; a dimension's spread is the serial f32 sum of
// (v - c)^2 in data order (src/tsvq.rs:86-98), which no reordering may touch; the
// split dimension is the last of equal maxima (max_by, 101-105); the median is taken from the sorted values (108-116); the
// partition is stable (119-122); children exist only when both sides are non-empty (127-141).
//
// The levels follow each other without the host: the device numbers the children and lays out the next level, the host
// launches for as many nodes as the level can have and surplus CTAs leave at once.  Per level: centroids and spreads (one warp per
// node and 32 dimensions where nodes have fewer than 150 rows, a CTA up to 2048; chunk sums, a CTA per 1024 rows, means and a streaming kernel
// above), split_kernel (split
// dimension, keys, median by radix selection, stable partition; one cluster of CTAs per node), next_level_kernel.  A full
// 64-bit sort of all rows per level, and two round trips to the host, took 0.16 + 0.08 ms of the 0.39 ms of a level of 100,000 x 128.
// The build is not sharded: every rank of a multi-GPU job builds the same tree.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstdlib>
#include <vector>

#include "cuda_device.hpp"
#include "kernels_common.cuh"
#include "row_walk.cuh"
#include "tsvq.hpp"
#include "umma.cuh"

namespace vqb {

namespace {

struct NodeInfo {
    unsigned int start, count; // positions of its rows in perm
    unsigned int chunk0, nchunks; // its 1024-row chunks in the level's chunk table
    unsigned int nleft;
    int split; // 1: this node is being split at this level
};

// What the host does not know of a level: written by next_level_kernel for the level after it.
struct LevelInfo {
    int first, count; // its nodes
    int chunks;
    int splits;       // nodes of it that are being split
};

constexpr unsigned MEAN_CHUNK = 1024;
struct ChunkInfo {
    unsigned int start, rows; // position of the chunk's first row in perm
};

constexpr uint32_t DEAD = 0xFFFFFFFFu;

// order-preserving map of f32 onto u32 (no NaN here)
__device__ __forceinline__ uint32_t f32_key(float v)
{
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_f32(uint32_t k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7FFFFFFFu) : ~k);
}

constexpr int WR_WARPS = 2; // warps per CTA of the kernels that walk rows (16 KiB of ring each)

__global__ void init_tree_kernel(size_t n, int splits, uint32_t *perm, NodeInfo *nodes, ChunkInfo *chunks, LevelInfo *level)
{
    after_previous_kernel();
    next_kernel_may_start();
    const size_t nchunks = (n + MEAN_CHUNK - 1) / MEAN_CHUNK;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        perm[i] = (uint32_t)i;
        if (i < nchunks) chunks[i] = ChunkInfo{(unsigned)(i * MEAN_CHUNK), (unsigned)min((size_t)MEAN_CHUNK, n - i * MEAN_CHUNK)};
        if (i == 0) {
            nodes[0] = NodeInfo{0u, (unsigned)n, 0u, (unsigned)nchunks, 0u, splits};
            level[0] = LevelInfo{0, 1, (int)nchunks, splits};
        }
    }
}

// ---- large nodes: one CTA per (1024-row chunk, 32 dimensions), then one thread per (node, dimension) adds the node's chunk
// sums in order and divides
template <bool VEC>
__global__ void __launch_bounds__(STREAM_THREADS) chunk_sums_kernel(const float *__restrict__ x, size_t dim, const uint32_t *perm,
                                                                    const LevelInfo *level, const ChunkInfo *chunks, float *partial)
{
    extern __shared__ __align__(16) float ring[];
    after_previous_kernel();
    next_kernel_may_start();
    const size_t groups = (dim + 31) / 32, chunk = blockIdx.x / groups, d0 = blockIdx.x % groups * 32, d = d0 + (threadIdx.x & 31);
    if (chunk >= (size_t)level->chunks) return;
    const ChunkInfo ch = chunks[chunk];
    float acc = 0.0f;
    stream_rows<VEC>(ring, x + d0, dim, perm + ch.start, ch.rows, (int)min(dim - d0, (size_t)32), [&](float v) { acc = __fadd_rn(acc, v); }, [](uint32_t) {});
    if (threadIdx.x >= 32 * STREAM_PRODUCERS && d < dim) partial[chunk * dim + d] = acc;
}

__global__ void node_mean_kernel(const NodeInfo *nodes, const LevelInfo *level, size_t dim, const float *partial, float *centroids)
{
    after_previous_kernel();
    next_kernel_may_start();
    const size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (t >= (size_t)level->count * dim) return;
    const int node = level->first + (int)(t / dim);
    const size_t d = t % dim;
    const NodeInfo nd = nodes[node];
    float total = 0.0f;
    const float *p = partial + (size_t)nd.chunk0 * dim + d;
#pragma unroll 8
    for (unsigned c = 0; c < nd.nchunks; ++c) total = __fadd_rn(total, p[(size_t)c * dim]);
    centroids[(size_t)node * dim + d] = __fdiv_rn(total, __uint2float_rn(nd.count)); // sum / (len as f32)
}

// ---- one warp per (node, 32 dimensions): the node's mean (MEAN: the sums of its 1024-row chunks one after the other) and, if
// it is going to be split, its spread
template <bool VEC>
__global__ void __launch_bounds__(32 * WR_WARPS) node_stats_kernel(const float *__restrict__ x, size_t dim, const uint32_t *perm,
                                                                   const NodeInfo *nodes, const LevelInfo *level, float *centroids, float *spread)
{
    __shared__ __align__(16) WalkRing ring[WR_WARPS];
    after_previous_kernel();
    next_kernel_may_start();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t groups = (dim + 31) / 32, unit = (size_t)blockIdx.x * WR_WARPS + warp;
    const size_t in_level = unit / groups, d0 = unit % groups * 32, d = d0 + lane;
    if (in_level >= (size_t)level->count) return;
    const int node = level->first + (int)in_level;
    const NodeInfo nd = nodes[node];
    const bool live = d < dim;
    const int cols = (int)min(dim - d0, (size_t)32);
    const uint32_t *rows = perm + nd.start;
    float total = 0.0f;
    for (unsigned r = 0; r < nd.count; r += MEAN_CHUNK) {
        float acc = 0.0f;
        walk_rows<32, VEC>(ring[warp], x + d0, dim, rows + r, min(MEAN_CHUNK, nd.count - r), cols, [&](float v) { acc = __fadd_rn(acc, v); });
        total = __fadd_rn(total, acc);
    }
    const float c = __fdiv_rn(total, __uint2float_rn(nd.count));
    if (live) centroids[(size_t)node * dim + d] = c;
    if (!nd.split) return;
    float var = 0.0f;
    walk_rows<32, VEC>(ring[warp], x + d0, dim, rows, nd.count, cols, [&](float v) {
        const float e = __fsub_rn(v, c);
        var = __fadd_rn(var, __fmul_rn(e, e));
    });
    if (live) spread[in_level * dim + d] = var;
}

// The same by a CTA per (node, 32 dimensions).
template <bool VEC>
__global__ void __launch_bounds__(STREAM_THREADS) node_stats_stream_kernel(const float *__restrict__ x, size_t dim, const uint32_t *perm,
                                                                           const NodeInfo *nodes, const LevelInfo *level, float *centroids, float *spread)
{
    extern __shared__ __align__(16) float ring[];
    after_previous_kernel();
    next_kernel_may_start();
    const size_t groups = (dim + 31) / 32, in_level = blockIdx.x / groups, d0 = blockIdx.x % groups * 32, d = d0 + (threadIdx.x & 31);
    if (in_level >= (size_t)level->count) return;
    const int node = level->first + (int)in_level;
    const NodeInfo nd = nodes[node];
    const bool live = threadIdx.x >= 32 * STREAM_PRODUCERS && d < dim;
    const int cols = (int)min(dim - d0, (size_t)32);
    const uint32_t *rows = perm + nd.start;
    static_assert(MEAN_CHUNK % STREAM_STAGE == 0, "a chunk's sum ends with a stage");
    float total = 0.0f, acc = 0.0f;
    const uint32_t last = (nd.count + STREAM_STAGE - 1) / STREAM_STAGE - 1;
    stream_rows<VEC>(ring, x + d0, dim, rows, nd.count, cols, [&](float v) { acc = __fadd_rn(acc, v); }, [&](uint32_t t) {
        if (t == last || (t + 1) % (MEAN_CHUNK / STREAM_STAGE) == 0) total = __fadd_rn(total, acc), acc = 0.0f;
    });
    const float c = __fdiv_rn(total, __uint2float_rn(nd.count));
    if (live) centroids[(size_t)node * dim + d] = c;
    if (!nd.split) return;
    float var = 0.0f;
    stream_rows<VEC>(ring, x + d0, dim, rows, nd.count, cols, [&](float v) {
        const float e = __fsub_rn(v, c);
        var = __fadd_rn(var, __fmul_rn(e, e));
    }, [](uint32_t) {});
    if (live) spread[in_level * dim + d] = var;
}

// ---- spreads of large nodes.  The sum stays one serial f32 chain per (node, dimension) in data order -- a dependent addition every
// 4.1 cycles at best, 5.0 here (root of 100,000 x 128: 258 us) -- so the kernel's job is to keep that chain fed: one CTA per
// (node, 32 dimensions); warp 0 is the consumer (lane = dimension, alone on its scheduler) and does nothing but read stages from
// shared memory and add; twelve producer warps on the other three schedulers gather the node's rows (128-bit loads where rows are
// whole 16-byte pieces (VEC), else four 32-bit ones, which still meet the chain's pace; 64 rows per warp in flight, the next
// stage's row numbers requested meanwhile), form (v - c)^2 with each term rounded like the reference's (src/tsvq.rs:86-98) and
// store that into a ring of 64-row stages, so the consumer's work per row is a quarter of a shared-memory load and one addition.
//
// A stage is stored dimension-major, [32 dimensions][64 rows], so that the consumer fetches four consecutive rows of its
// dimension with one 128-bit load; the 16 four-row groups of a dimension are permuted by ns_swizzle(d), which keeps both
// the producers' 32-bit stores and the consumer's 128-bit loads free of bank conflicts.
//
// Hand-over.  A poll of an mbarrier costs the consumer 230 cycles even when the phase is complete (the instruction that
// reads the poll's predicate stalls the warp until the answer is back), as much as the 64 additions of a stage.  So the
// producers announce finished stages with a shared-memory counter per group of four stages, which the consumer reads
// with an ordinary load one group ahead -- the load is in flight during the additions and is looked at three stages
// later -- and the consumer hands a group back with one relaxed arrive.  Stage numbers are padded to a multiple of four
// (padding stages are announced without data) so that every group sees exactly four announcements.
constexpr int NS_STAGE_ROWS = 64, NS_GROUP = 4, NS_GROUPS = 6, NS_RING = NS_GROUP * NS_GROUPS, NS_PRODUCERS = 12, NS_THREADS = 512;
constexpr int NS_STAGE_BYTES = NS_STAGE_ROWS * 128;
constexpr int NS_SMEM = NS_RING * NS_STAGE_BYTES + NS_GROUPS * 8 + NS_GROUPS * 4;
// a producer may wait for the release of a group only when the release before that one has certainly happened (a parity
// wait cannot tell two phases apart); the same warp filled a stage NS_PRODUCERS stages earlier, so this holds while
// NS_PRODUCERS <= NS_RING - NS_GROUP
static_assert(NS_PRODUCERS <= NS_RING - NS_GROUP, "parity waits need the producers' lead to stay inside the ring");
constexpr int NS_ERR_WAIT = 190;
constexpr uint32_t NS_SPIN_LIMIT = 1u << 28;

__device__ __forceinline__ int ns_swizzle(int d) { return ((d & 7) ^ (d >> 3)) & 7; }

template <bool VEC>
__global__ void __launch_bounds__(NS_THREADS) node_spread_stream_kernel(const float *__restrict__ x, size_t dim, const uint32_t *__restrict__ perm,
                                                                        const NodeInfo *nodes, const LevelInfo *level, const float *centroids, float *spread, int *error)
{
    extern __shared__ __align__(256) unsigned char ns_smem[];
    float *ring = reinterpret_cast<float *>(ns_smem);
    uint64_t *empty = reinterpret_cast<uint64_t *>(ns_smem + NS_RING * NS_STAGE_BYTES);
    volatile uint32_t *filled = reinterpret_cast<volatile uint32_t *>(empty + NS_GROUPS);
    __shared__ int abort_flag;
    after_previous_kernel();
    next_kernel_may_start();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned groups = (unsigned)((dim + 31) / 32), in_level = blockIdx.x / groups;
    if (in_level >= (unsigned)level->count) return;
    const int node = level->first + (int)in_level;
    const NodeInfo nd = nodes[node];
    if (!nd.split) return;
    const size_t col0 = (size_t)(blockIdx.x % groups) * 32;
    const unsigned long long count = nd.count;
    const uint32_t S = (uint32_t)((count + NS_STAGE_ROWS - 1) / NS_STAGE_ROWS);      // stages with rows
    const uint32_t total = (S + NS_GROUP - 1) / NS_GROUP * NS_GROUP;                   // stage numbers
    if (threadIdx.x == 0) {
        for (int i = 0; i < NS_GROUPS; ++i) mbar_init(&empty[i], 1), filled[i] = 0;
        abort_flag = 0;
    }
    __syncthreads();
    if (warp == 0) {
        float4 a[8], b[8];
        float acc = 0.0f;
        bool ok = true;
        const int g = ns_swizzle(lane);
        auto group_ready = [&](uint32_t slot, uint32_t need, uint32_t have) { // have: filled[slot] as read a while ago
            if (have < need) {
                uint32_t i = 0;
                while (filled[slot] < need) {
                    if (++i >= NS_SPIN_LIMIT || ((i & 4095u) == 0 && *(volatile int *)&abort_flag)) {
                        if (i >= NS_SPIN_LIMIT) abort_flag = 1, atomicCAS(error, 0, NS_ERR_WAIT);
                        ok = false;
                        return;
                    }
                }
            }
            __threadfence_block(); // the stages' values are read after their announcement
        };
        // this lane's dimension in stage 0 of the ring: the four-row group q of its first (second) 32 rows sits at piece[q] (+ 128) bytes
        uint32_t piece[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) piece[q] = smem_u32(ring + lane * NS_STAGE_ROWS) + ((q ^ g) << 4);
        // volatile, so that the loads stay where they are written: between the additions, whose issue slots they fill
        auto load4 = [&](uint32_t at, int q) {
            float4 r;
            asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(r.x), "=f"(r.y), "=f"(r.z), "=f"(r.w) : "r"(at + piece[q]));
            return r;
        };
        auto request = [&](uint32_t s, float4(&buf)[16]) {
#pragma unroll
            for (int q = 0; q < 16; ++q) buf[q] = load4((s % NS_RING) * NS_STAGE_BYTES, q);
        };
        // adds the 32 rows in cur and loads the ones at byte `at` of the ring: the loads among the first half of the additions, so
        // that the second half covers their latency
        auto half_stage = [&](float4(&cur)[8], float4(&nxt)[8], uint32_t at) {
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (q < 4) nxt[2 * q] = load4(at, 2 * q), nxt[2 * q + 1] = load4(at, 2 * q + 1);
                acc = __fadd_rn(acc, cur[q].x), acc = __fadd_rn(acc, cur[q].y);
                acc = __fadd_rn(acc, cur[q].z), acc = __fadd_rn(acc, cur[q].w);
            }
        };
        group_ready(0, NS_GROUP, 0);
        if (ok) {
#pragma unroll
            for (int q = 0; q < 8; ++q) a[q] = load4(0, q);
        }
        // Groups with another one behind them (their stages are full) run without a branch but the loop's: tests and addresses computed
        // per stage took 240 cycles beside the 280 of its 64 additions (100,000 rows: 462 -> 310 us).
        uint32_t at = 0, slot = 0, need = NS_GROUP, s = 0;
        for (; ok && s + NS_GROUP < S; s += NS_GROUP) {
            const uint32_t next_slot = slot + 1 == NS_GROUPS ? 0 : slot + 1, next = next_slot * (NS_GROUP * NS_STAGE_BYTES);
            if (next_slot == 0) need += NS_GROUP;
            const uint32_t have = filled[next_slot];
#pragma unroll
            for (int i = 0; i < NS_GROUP - 1; ++i) {
                half_stage(a, b, at + i * NS_STAGE_BYTES + 128);
                half_stage(b, a, at + (i + 1) * NS_STAGE_BYTES);
            }
            half_stage(a, b, at + (NS_GROUP - 1) * NS_STAGE_BYTES + 128);
            group_ready(next_slot, need, have);
            if (!ok) break;
            half_stage(b, a, next);
            __syncwarp(); // every lane has used its values
            if (lane == 0) mbar_arrive_relaxed(&empty[slot]);
            at = next, slot = next_slot;
        }
        for (; ok && s < S; ++s, at += NS_STAGE_BYTES) { // the last group; nobody waits for its return
            const uint32_t left = (uint32_t)(count - (unsigned long long)s * NS_STAGE_ROWS);
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                const float4 v = load4(at + (q >> 3) * 128, q & 7);
                if (4 * q + 0 < left) acc = __fadd_rn(acc, v.x);
                if (4 * q + 1 < left) acc = __fadd_rn(acc, v.y);
                if (4 * q + 2 < left) acc = __fadd_rn(acc, v.z);
                if (4 * q + 3 < left) acc = __fadd_rn(acc, v.w);
            }
        }
        if (ok && col0 + lane < dim) spread[(size_t)in_level * dim + col0 + lane] = acc;
    } else if ((warp & 3) != 0) {
        const uint32_t *rows = perm + nd.start;
        const int sub = lane >> 3, piece = lane & 7;
        const float *xcol = x + col0 + piece * 4;
        const uint32_t ld = (uint32_t)dim;
        const int live = (int)min((unsigned long long)4, dim > col0 + piece * 4 ? (unsigned long long)(dim - (col0 + piece * 4)) : 0ull); // this lane's columns
        auto load_piece = [&](const float *p) {
            float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
            if (VEC) {
                if (live) r = __ldg(reinterpret_cast<const float4 *>(p));
            } else {
                if (live > 0) r.x = __ldg(p);
                if (live > 1) r.y = __ldg(p + 1);
                if (live > 2) r.z = __ldg(p + 2);
                if (live > 3) r.w = __ldg(p + 3);
            }
            return r;
        };
        float4 cc = make_float4(0.f, 0.f, 0.f, 0.f); // (node_mean_kernel may have written it while this kernel was already there: ordinary loads)
        {
            const float *c = centroids + (size_t)node * dim + col0 + piece * 4;
            if (live > 0) cc.x = c[0];
            if (live > 1) cc.y = c[1];
            if (live > 2) cc.z = c[2];
            if (live > 3) cc.w = c[3];
        }
        // this lane's four dimensions 4 * piece + j, row position sub: a stage begins on 256 bytes, so the four-row group i lies at the
        // address of group 0 with i exchanged into bits 4 to 7
        uint32_t dst[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[j] = smem_u32(ring + (4 * piece + j) * NS_STAGE_ROWS + sub) + (ns_swizzle(4 * piece + j) << 4);
        uint32_t idx[16];
        auto load_idx = [&](uint32_t s) { // stage numbers past the node's rows give no rows at all
            const uint32_t left = s < S ? (uint32_t)count - s * NS_STAGE_ROWS : 0u;
            const uint32_t *p = rows + (size_t)s * NS_STAGE_ROWS + sub;
#pragma unroll
            for (int i = 0; i < 16; ++i) idx[i] = 4 * i + sub < left ? p[4 * i] : DEAD;
        };
        auto load_rows = [&](float4(&v)[16]) {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                v[i] = idx[i] != DEAD ? load_piece(xcol + (unsigned long long)idx[i] * ld) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        auto put = [&](float4(&v)[16], uint32_t s) { // false: a wait ran out
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                float d;
                d = __fsub_rn(v[i].x, cc.x), v[i].x = __fmul_rn(d, d);
                d = __fsub_rn(v[i].y, cc.y), v[i].y = __fmul_rn(d, d);
                d = __fsub_rn(v[i].z, cc.z), v[i].z = __fmul_rn(d, d);
                d = __fsub_rn(v[i].w, cc.w), v[i].w = __fmul_rn(d, d);
            }
            const uint32_t grp = s / NS_GROUP, gslot = grp % NS_GROUPS;
            if (!mbar_wait<100u>(&empty[gslot], ((grp / NS_GROUPS) & 1u) ^ 1u, &abort_flag, error, NS_ERR_WAIT)) return false;
            if (s < S) { // not padding
                const uint32_t at = s % NS_RING * NS_STAGE_BYTES;
                auto store = [&](int j, int i, float value) {
                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(((at + dst[j]) ^ ((i & 7) << 4)) + (i >> 3) * 128), "f"(value) : "memory");
                };
#pragma unroll
                for (int i = 0; i < 16; ++i) store(0, i, v[i].x), store(1, i, v[i].y), store(2, i, v[i].z), store(3, i, v[i].w);
            }
            __syncwarp();
            if (lane == 0) {
                __threadfence_block(); // the stage's values before its announcement
                atomicAdd(const_cast<uint32_t *>(&filled[gslot]), 1u);
            }
            return true;
        };
        float4 v[16];
        uint32_t s = (warp >> 2) * 3 + (warp & 3) - 1;
        load_idx(s);
        for (; s < total; s += NS_PRODUCERS) {
            load_rows(v);
            load_idx(s + NS_PRODUCERS);
            if (!put(v, s)) break;
        }
    }
}

// Everything between a node's spreads and its two halves, one cluster of CTAs per node (one CTA where the level's nodes are
// small): the split dimension (last of equal maxima), the rows' values along it as ordered keys, the element of rank count / 2 by
// radix selection (11 + 11 + 10 bits; the CTAs add up their digit counts through distributed shared memory), for an even
// count its predecessor, the median, and the stable partition.
constexpr int SP_THREADS = 512, SP_BINS = 2048, SP_CLUSTER = 8;
constexpr unsigned SP_KEYS = 16384; // keys that a CTA keeps in shared memory
constexpr int SP_U = 8;             // loads of a thread in flight
constexpr int SP_RUN = 4;           // rows of a thread at a time in the partition

__global__ void __launch_bounds__(SP_THREADS) split_kernel(const float *__restrict__ x, size_t dim, const uint32_t *__restrict__ perm, uint32_t *perm_out,
                                                           NodeInfo *nodes, const LevelInfo *level, const float *spread, uint32_t *keys, unsigned room, int *error)
{
    after_previous_kernel();
    next_kernel_may_start();
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    const unsigned cs = cl.num_blocks(), rank = cl.block_rank();
    const unsigned in_level = blockIdx.x / cs;
    if (in_level >= (unsigned)level->count) return; // the whole cluster leaves
    const int node = level->first + (int)in_level;
    const NodeInfo nd = nodes[node];
    if (!nd.split) return;
    extern __shared__ uint32_t s_keys[];
    __shared__ __align__(16) uint32_t s_hist[SP_BINS];
    __shared__ uint32_t s_scan[SP_THREADS / 32], s_bin, s_below, s_left, s_max;
    __shared__ unsigned long long s_best;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) s_best = 0ull, s_left = 0u, s_max = 0u;
    __syncthreads();
    {
        unsigned long long best = 0ull;
        for (size_t t = tid; t < dim; t += SP_THREADS) {
            const float v = spread[(size_t)in_level * dim + t];
            if (!(v == v)) atomicExch(error, 105); // not comparable
            const unsigned long long key = ((unsigned long long)f32_key(v) << 32) | (unsigned)t;
            best = key > best ? key : best;
        }
        atomicMax(&s_best, best);
    }
    __syncthreads();
    const size_t split_dim = min((size_t)(uint32_t)s_best, dim - 1);

    const unsigned per = (nd.count + cs - 1) / cs, r0 = min(nd.count, rank * per), r1 = min(nd.count, r0 + per);
    const uint32_t *rows = perm + nd.start;
    // f(key of row i) for this CTA's rows, several of a thread's keys on their way at once where they are in memory
    uint32_t *const far_keys = keys + nd.start;
    const bool fits = r1 - r0 <= room;
    auto for_keys = [&](auto f) {
        if (fits) {
#pragma unroll 4
            for (unsigned i = r0 + tid; i < r1; i += SP_THREADS) f(s_keys[i - r0]);
        } else {
            for (unsigned i0 = r0 + tid; i0 < r1; i0 += SP_U * SP_THREADS) {
                uint32_t key[SP_U];
#pragma unroll
                for (int u = 0; u < SP_U; ++u) key[u] = i0 + u * SP_THREADS < r1 ? far_keys[i0 + u * SP_THREADS] : 0u;
#pragma unroll
                for (int u = 0; u < SP_U; ++u)
                    if (i0 + u * SP_THREADS < r1) f(key[u]);
            }
        }
    };
    auto meet = [&] { // all CTAs of the node
        if (cs > 1) cl.sync();
        else __syncthreads();
    };
    bool nan = false;
    for (unsigned i0 = r0 + tid; i0 < r1; i0 += SP_U * SP_THREADS) {
        uint32_t row[SP_U];
        float v[SP_U];
#pragma unroll
        for (int u = 0; u < SP_U; ++u) row[u] = i0 + u * SP_THREADS < r1 ? rows[i0 + u * SP_THREADS] : 0u;
#pragma unroll
        for (int u = 0; u < SP_U; ++u) v[u] = i0 + u * SP_THREADS < r1 ? __ldg(x + (size_t)row[u] * dim + split_dim) : 0.0f;
#pragma unroll
        for (int u = 0; u < SP_U; ++u) {
            const unsigned i = i0 + u * SP_THREADS;
            nan = nan || !(v[u] == v[u]);
            if (i < r1) (fits ? s_keys[i - r0] : far_keys[i]) = f32_key(v[u]);
        }
    }
    if (nan) atomicExch(error, 105);
    __syncthreads(); // from here on a CTA reads the keys of its own rows only

    // inclusive scan of one value per thread; the CTA's total in s_scan[last]
    auto block_scan = [&](uint32_t v) {
        uint32_t incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        __syncthreads();
        if (lane == 31) s_scan[warp] = incl;
        __syncthreads();
        if (warp == 0) {
            uint32_t w = lane < SP_THREADS / 32 ? s_scan[lane] : 0u;
#pragma unroll
            for (int o = 1; o < SP_THREADS / 32; o <<= 1) {
                const uint32_t up = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += up;
            }
            if (lane < SP_THREADS / 32) s_scan[lane] = w;
        }
        __syncthreads();
        return incl + (warp ? s_scan[warp - 1] : 0u);
    };

    uint32_t r = nd.count / 2, prefix = 0u, mask = 0u;
#pragma unroll 1
    for (int pass = 0; pass < 3; ++pass) {
        const int shift = pass == 0 ? 21 : pass == 1 ? 10 : 0;
        const uint32_t digit = pass == 2 ? 1023u : 2047u;
        for (int b = tid; b < SP_BINS; b += SP_THREADS) s_hist[b] = 0u;
        __syncthreads();
        for_keys([&](uint32_t key) {
            if ((key & mask) == prefix) atomicAdd(s_hist + ((key >> shift) & digit), 1u);
        });
        meet();
        uint32_t c[SP_BINS / SP_THREADS], sum = 0u;
#pragma unroll
        for (int b = 0; b < SP_BINS / SP_THREADS; ++b) c[b] = 0u;
        for (unsigned q = 0; q < cs; ++q) {
            const uint4 h = *reinterpret_cast<const uint4 *>(cl.map_shared_rank(s_hist, q) + 4 * tid);
            c[0] += h.x, c[1] += h.y, c[2] += h.z, c[3] += h.w;
        }
#pragma unroll
        for (int b = 0; b < SP_BINS / SP_THREADS; ++b) sum += c[b];
        uint32_t below = block_scan(sum) - sum;
#pragma unroll
        for (int b = 0; b < SP_BINS / SP_THREADS; ++b) {
            if (r >= below && r - below < c[b]) s_bin = 4 * tid + b, s_below = below;
            below += c[b];
        }
        meet(); // the counts have been read everywhere before they are cleared
        prefix |= s_bin << shift, mask |= digit << shift;
        r -= s_below;
    }
    const float hi = key_f32(prefix);
    float median = hi;
    if (nd.count % 2 == 0) {
        float lo = hi; // r > 0: the predecessor equals it
        if (r == 0) {  // (the same in every CTA)
            uint32_t low = 0u;
            for_keys([&](uint32_t key) {
                if (key < prefix) low = max(low, key);
            });
            low = __reduce_max_sync(0xffffffffu, low);
            if (lane == 0) atomicMax(&s_max, low);
            meet();
            low = 0u;
            for (unsigned q = 0; q < cs; ++q) low = max(low, *cl.map_shared_rank(&s_max, q));
            lo = key_f32(low);
        }
        median = __fdiv_rn(__fadd_rn(lo, hi), 2.0f);
    }

    // stable partition: the rows at or below the median first, both sides in their old order
    uint32_t mine = 0u;
    for_keys([&](uint32_t key) { mine += key_f32(key) <= median ? 1u : 0u; });
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) atomicAdd(&s_left, mine);
    meet();
    uint32_t before = 0u, nleft = 0u;
    for (unsigned q = 0; q < cs; ++q) {
        const uint32_t l = *cl.map_shared_rank(&s_left, q);
        before += q < rank ? l : 0u;
        nleft += l;
    }
    meet(); // nobody leaves while its shared memory is still being read
    // a thread takes SP_RUN rows in a row, so that the scan is needed once for SP_RUN * SP_THREADS of them
    for (unsigned t0 = r0; t0 < r1; t0 += SP_RUN * SP_THREADS) {
        const unsigned i0 = t0 + SP_RUN * tid;
        uint32_t row[SP_RUN], lefts = 0u;
        bool left[SP_RUN];
#pragma unroll
        for (int u = 0; u < SP_RUN; ++u) {
            const bool in = i0 + u < r1;
            row[u] = in ? rows[i0 + u] : 0u;
            left[u] = in && key_f32(fits ? s_keys[i0 + u - r0] : far_keys[i0 + u]) <= median;
            lefts += left[u] ? 1u : 0u;
        }
        uint32_t at = before + block_scan(lefts) - lefts;
#pragma unroll
        for (int u = 0; u < SP_RUN; ++u) {
            if (i0 + u < r1) perm_out[nd.start + (left[u] ? at : nleft + (i0 + u - at))] = row[u];
            at += left[u] ? 1u : 0u;
        }
        before += s_scan[SP_THREADS / 32 - 1];
        // (block_scan's first barrier keeps s_scan until everybody has read the total)
    }
    if (rank == 0 && tid == 0) nodes[node].nleft = nleft;
}

// Numbers the children of a level in order (both or none, src/tsvq.rs:127-141), lays them and their chunks out for the next one.
__global__ void __launch_bounds__(1024) next_level_kernel(NodeInfo *nodes, const LevelInfo *level, LevelInfo *next, int may_split, int32_t *left, int32_t *right,
                                                          ChunkInfo *chunks)
{
    __shared__ unsigned long long s_scan[32], s_carry;
    __shared__ int s_splits;
    after_previous_kernel();
    next_kernel_may_start();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const LevelInfo li = *level;
    if (tid == 0) s_carry = 0ull, s_splits = 0;
    __syncthreads();
    for (int t0 = 0; t0 < li.count; t0 += 1024) {
        const int node = li.first + t0 + tid;
        const bool in = t0 + tid < li.count;
        NodeInfo nd = {};
        if (in) nd = nodes[node];
        const bool has = in && nd.split && nd.nleft > 0 && nd.nleft < nd.count;
        const unsigned nl = nd.nleft, nr = nd.count - nl;
        const unsigned cl = (nl + MEAN_CHUNK - 1) / MEAN_CHUNK, cr = (nr + MEAN_CHUNK - 1) / MEAN_CHUNK;
        // pairs of children in the low, their chunks in the high half
        const unsigned long long mine = has ? ((unsigned long long)(cl + cr) << 32) | 1ull : 0ull;
        unsigned long long incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned long long up = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += up;
        }
        if (lane == 31) s_scan[warp] = incl;
        __syncthreads();
        unsigned long long at = s_carry + incl - mine;
        for (int w = 0; w < warp; ++w) at += s_scan[w];
        if (in) {
            int l = -1, r = -1;
            if (has) {
                l = li.first + li.count + 2 * (int)(uint32_t)at, r = l + 1;
                const unsigned c0 = (unsigned)(at >> 32);
                const NodeInfo a = {nd.start, nl, c0, cl, 0u, may_split && nl > 1 ? 1 : 0}, b = {nd.start + nl, nr, c0 + cl, cr, 0u, may_split && nr > 1 ? 1 : 0};
                nodes[l] = a, nodes[r] = b;
                for (unsigned c = 0; c < cl; ++c) chunks[c0 + c] = ChunkInfo{a.start + c * MEAN_CHUNK, min(MEAN_CHUNK, nl - c * MEAN_CHUNK)};
                for (unsigned c = 0; c < cr; ++c) chunks[c0 + cl + c] = ChunkInfo{b.start + c * MEAN_CHUNK, min(MEAN_CHUNK, nr - c * MEAN_CHUNK)};
                if (a.split + b.split) atomicAdd(&s_splits, a.split + b.split);
            }
            left[node] = l, right[node] = r;
        }
        __syncthreads();
        if (tid == 1023) s_carry = at + mine;
        __syncthreads();
    }
    if (tid == 0) *next = LevelInfo{li.first + li.count, 2 * (int)(uint32_t)s_carry, (int)(s_carry >> 32), s_splits};
}

__global__ void no_children_kernel(const LevelInfo *level, int32_t *left, int32_t *right) // of the deepest level
{
    after_previous_kernel();
    next_kernel_may_start();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < level->count) left[level->first + t] = right[level->first + t] = -1;
}

template <int METRIC>
__global__ void tsvq_quantize_kernel(const float *x, size_t n, size_t dim, const float *centroids, const int32_t *left, const int32_t *right, float pv,
                                     uint16_t *out_f16, uint32_t *leaf_out)
{
    for (size_t row = blockIdx.x * (size_t)blockDim.x + threadIdx.x; row < n; row += (size_t)gridDim.x * blockDim.x) {
        const float *v = x + row * dim;
        float norm_a = 0.0f;
        if (METRIC == M_COSINE) norm_a = norm_chain(v, (int)dim, 1);
        int node = 0;
        for (;;) {
            const int l = left[node], r = right[node];
            if (l >= 0 && r >= 0) {
                const float *cl = centroids + (size_t)l * dim, *cr = centroids + (size_t)r * dim;
                DistAcc<METRIC> al, ar;
                al.init();
                ar.init();
                for (size_t t = 0; t < dim; ++t) {
                    const float xv = v[t];
                    al.step(xv, cl[t], pv);
                    ar.step(xv, cr[t], pv);
                }
                const float dl = al.finish(pv, norm_a), dr = ar.finish(pv, norm_a);
                node = (dl <= dr) ? l : r; // src/tsvq.rs:172: the left child on ties; a NaN distance sends the row right
            } else if (l >= 0) {
                node = l;
            } else if (r >= 0) {
                node = r;
            } else {
                break;
            }
        }
        if (leaf_out) leaf_out[row] = (uint32_t)node;
        if (out_f16) {
            const float *c = centroids + (size_t)node * dim;
            for (size_t t = 0; t < dim; ++t) out_f16[row * dim + t] = f32_to_f16_bits(c[t]);
        }
    }
}

// The lookup for the Euclidean metrics, rows of up to 256 dimensions: eight lanes per row, four rows per warp.  The row stays in
// registers; at each node the lanes add up their shares of both children's squared distances, and the smaller one wins where
// the two differ by more than any order of summation could explain.  The serial chain that the reference evaluates (src/tsvq.rs:
// 159-175) is only walked where they do not, or where values overflow, vanish or are NaN.
//
// Bound: all terms are >= 0, so a sum of dim of them carries a relative error of at most (dim + 2) u in either order (u = 2^-24; a
// term's own three roundings included), and the square roots of two numbers further apart than 4 u keep their order.  Twice
// (dim + 2) u + 4 u is well below the (4 dim + 64) u that is asked for.
//
// One thread per row reads 16 bytes of 32 different nodes per load: 32 wavefronts where this takes four.  1M x 64, depth 6: 505 -> 241 us;
// 1M x 127, depth 8: 3070 -> 878 us; one row of 128, depth 8: 34 -> 15 us with the call around it.
template <int METRIC, bool VEC, int NP>
__global__ void __launch_bounds__(256) tsvq_quantize_group_kernel(const float *__restrict__ x, size_t n, int dim, const float *__restrict__ centroids,
                                                                  const int32_t *__restrict__ left, const int32_t *__restrict__ right, float pv,
                                                                  uint16_t *out_f16, uint32_t *leaf_out)
{
    const int lane = threadIdx.x & 31, sub = lane & 7, group = lane >> 3;
    const float eps = (4.0f * dim + 64.0f) * 5.9604645e-8f;
    // the lane's q-th share of a row: VEC: columns 4 (sub + 8 q) + e, else sub + 8 (4 q + e)
    auto load = [&](const float *row, float(&v)[NP][4]) {
#pragma unroll
        for (int q = 0; q < NP; ++q) {
            if (VEC) {
                float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                if (4 * (sub + 8 * q) < dim) f = __ldg(reinterpret_cast<const float4 *>(row) + sub + 8 * q);
                v[q][0] = f.x, v[q][1] = f.y, v[q][2] = f.z, v[q][3] = f.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) v[q][e] = sub + 8 * (4 * q + e) < dim ? __ldg(row + sub + 8 * (4 * q + e)) : 0.0f;
            }
        }
    };
    const size_t warps = (size_t)gridDim.x * (blockDim.x >> 5);
    for (size_t row0 = (blockIdx.x * (size_t)(blockDim.x >> 5) + (threadIdx.x >> 5)) * 4; row0 < n; row0 += warps * 4) {
        const size_t row = row0 + group;
        const bool there = row < n;
        const float *xr = x + (there ? row : n - 1) * dim;
        float v[NP][4];
        load(xr, v);
        int node = 0, l = there ? left[0] : -1, r = there ? right[0] : -1;
        while (__any_sync(0xffffffffu, l >= 0 || r >= 0)) {
            const bool both = l >= 0 && r >= 0;
            int ll = -1, lr = -1, rl = -1, rr = -1; // of the next level, on their way during the distances
            float sl = 0.0f, sr = 0.0f;
            if (both) {
                ll = left[l], lr = right[l], rl = left[r], rr = right[r];
                float a[NP][4], b[NP][4];
                load(centroids + (size_t)l * dim, a);
                load(centroids + (size_t)r * dim, b);
#pragma unroll
                for (int q = 0; q < NP; ++q)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float da = v[q][e] - a[q][e], db = v[q][e] - b[q][e];
                        sl = fmaf(da, da, sl), sr = fmaf(db, db, sr);
                    }
            }
#pragma unroll
            for (int o = 4; o; o >>= 1) sl += __shfl_xor_sync(0xffffffffu, sl, o), sr += __shfl_xor_sync(0xffffffffu, sr, o);
            if (both) {
                const float most = fmaxf(sl, sr);
                bool go_left = sl < sr;
                if (!(fabsf(sl - sr) > eps * most && most > 1e-25f && most < 1e37f)) { // the same in the row's eight lanes
                    const unsigned mates = 0xFFu << (8 * group);
                    float d = 0.0f;
                    if (sub < 2) {
                        const float *c = centroids + (size_t)(sub ? r : l) * dim;
                        DistAcc<METRIC> acc;
                        acc.init();
                        for (int t = 0; t < dim; ++t) acc.step(xr[t], c[t], pv);
                        d = acc.finish(pv, 0.0f);
                    }
                    const float dl = __shfl_sync(mates, d, 8 * group), dr = __shfl_sync(mates, d, 8 * group + 1);
                    go_left = dl <= dr; // src/tsvq.rs:172: the left child on ties; a NaN distance sends the row right
                }
                node = go_left ? l : r;
                l = go_left ? ll : rl, r = go_left ? lr : rr;
            } else if (l >= 0 || r >= 0) {
                node = l >= 0 ? l : r;
                l = left[node], r = right[node];
            }
        }
        if (!there) continue; // no shuffle follows in this turn, and the next turn's are reached by all or by none
        if (leaf_out && sub == 0) leaf_out[row] = (uint32_t)node;
        if (out_f16) {
            float c[NP][4];
            load(centroids + (size_t)node * dim, c);
#pragma unroll
            for (int q = 0; q < NP; ++q) {
                if (VEC) {
                    if (4 * (sub + 8 * q) < dim)
                        __stcs(reinterpret_cast<uint2 *>(out_f16 + row * dim) + sub + 8 * q,
                               make_uint2((uint32_t)f32_to_f16_bits(c[q][0]) | ((uint32_t)f32_to_f16_bits(c[q][1]) << 16),
                                          (uint32_t)f32_to_f16_bits(c[q][2]) | ((uint32_t)f32_to_f16_bits(c[q][3]) << 16)));
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (sub + 8 * (4 * q + e) < dim) out_f16[row * dim + sub + 8 * (4 * q + e)] = f32_to_f16_bits(c[q][e]);
                }
            }
        }
    }
}

// Tile variant of the lookup for rows in whole 16-byte pieces (dim a multiple of 8, aligned pointers): a CTA stages 128
// rows in shared memory with coalesced 128-bit loads (row stride dim + 4 floats, so the per-thread 128-bit reads of the
// walk are conflict-free), every thread walks the tree for its own row with the same serial distance chains as above but
// fetches both children's centroids 16 bytes at a time, and the f16 rows of the leaves are written by the whole CTA in
// 16-byte pieces.  One thread per row reading its row straight from global memory spends its time on 32 different lines
// per load instruction and 2-byte stores 2 * dim bytes apart.
constexpr int TQ_ROWS = 128;
template <int METRIC>
__global__ void __launch_bounds__(TQ_ROWS) tsvq_quantize_tile_kernel(const float *__restrict__ x, size_t n, int dim, const float *__restrict__ centroids,
                                                                     const int32_t *__restrict__ left, const int32_t *__restrict__ right, float pv,
                                                                     uint16_t *out_f16, uint32_t *leaf_out)
{
    extern __shared__ __align__(16) float tq_rows[];
    __shared__ int leaf_sh[TQ_ROWS];
    const int stride = dim + 4, chunks = dim / 4, octs = dim / 8;
    for (size_t tile = blockIdx.x; tile * TQ_ROWS < n; tile += gridDim.x) {
        const size_t row0 = tile * TQ_ROWS;
        const int rows = (int)(n - row0 < (size_t)TQ_ROWS ? n - row0 : (size_t)TQ_ROWS);
        __syncthreads(); // the previous tile's readers are done
        const float4 *src = reinterpret_cast<const float4 *>(x + row0 * dim);
        for (int i = threadIdx.x; i < rows * chunks; i += TQ_ROWS) {
            const int r = i / chunks, c = i - r * chunks;
            *reinterpret_cast<float4 *>(tq_rows + r * stride + 4 * c) = __ldcs(src + i);
        }
        __syncthreads();
        if ((int)threadIdx.x < rows) {
            const float *v = tq_rows + threadIdx.x * stride;
            float norm_a = 0.0f;
            if (METRIC == M_COSINE) norm_a = norm_chain(v, dim, 1);
            int node = 0;
            for (;;) {
                const int l = left[node], r = right[node];
                if (l >= 0 && r >= 0) {
                    const float4 *cl = reinterpret_cast<const float4 *>(centroids + (size_t)l * dim);
                    const float4 *cr = reinterpret_cast<const float4 *>(centroids + (size_t)r * dim);
                    DistAcc<METRIC> al, ar;
                    al.init();
                    ar.init();
#pragma unroll 2
                    for (int c = 0; c < chunks; ++c) {
                        const float4 xv = *reinterpret_cast<const float4 *>(v + 4 * c);
                        const float4 a = __ldg(cl + c), b = __ldg(cr + c);
                        al.step(xv.x, a.x, pv), ar.step(xv.x, b.x, pv);
                        al.step(xv.y, a.y, pv), ar.step(xv.y, b.y, pv);
                        al.step(xv.z, a.z, pv), ar.step(xv.z, b.z, pv);
                        al.step(xv.w, a.w, pv), ar.step(xv.w, b.w, pv);
                    }
                    const float dl = al.finish(pv, norm_a), dr = ar.finish(pv, norm_a);
                    node = (dl <= dr) ? l : r; // src/tsvq.rs:172: the left child on ties; a NaN distance sends the row right
                } else if (l >= 0) {
                    node = l;
                } else if (r >= 0) {
                    node = r;
                } else {
                    break;
                }
            }
            leaf_sh[threadIdx.x] = node;
            if (leaf_out) leaf_out[row0 + threadIdx.x] = (uint32_t)node;
        }
        __syncthreads();
        if (out_f16) {
            for (int i = threadIdx.x; i < rows * octs; i += TQ_ROWS) {
                const int r = i / octs, o = i - r * octs;
                const float4 *c = reinterpret_cast<const float4 *>(centroids + (size_t)leaf_sh[r] * dim) + 2 * o;
                const float4 p = __ldg(c), q = __ldg(c + 1);
                uint4 w;
                w.x = (uint32_t)f32_to_f16_bits(p.x) | ((uint32_t)f32_to_f16_bits(p.y) << 16);
                w.y = (uint32_t)f32_to_f16_bits(p.z) | ((uint32_t)f32_to_f16_bits(p.w) << 16);
                w.z = (uint32_t)f32_to_f16_bits(q.x) | ((uint32_t)f32_to_f16_bits(q.y) << 16);
                w.w = (uint32_t)f32_to_f16_bits(q.z) | ((uint32_t)f32_to_f16_bits(q.w) << 16);
                __stcs(reinterpret_cast<uint4 *>(out_f16 + (row0 + r) * dim + 8 * o), w);
            }
        }
    }
}

struct Pool { // device memory of one build: freed in stream order, also when something throws
    CudaDevice &dev;
    std::vector<void *> all;
    ~Pool()
    {
        for (void *p : all) dev.release(p);
    }
    template <typename T> T *get(size_t items)
    {
        all.push_back(dev.alloc(sizeof(T) * items));
        return static_cast<T *>(all.back());
    }
};

inline unsigned grid_for(size_t items, int threads, unsigned cap)
{
    return (unsigned)std::max<size_t>(1, std::min<size_t>((items + threads - 1) / threads, cap));
}

} // namespace

void tsvq_fit(CudaDevice &dev, const float *x, size_t n, size_t dim, size_t max_depth, TsvqTree &out)
{
    if (n == 0 || dim == 0) throw Error(1, "Empty input: at least one vector is required.");
    if (n >= 0x7FFFFFFFull) throw Error(103, "tsvq: more than 2^31 - 2 rows are not supported");
    cudaStream_t st = dev.stream();
    const size_t cap_nodes = std::min<size_t>(max_depth < 40 ? ((size_t)2 << max_depth) - 1 : 2 * n, 2 * n);
    // A level's nodes are "small" when they average at most this many rows: one warp then walks mean and spread in about 12 cycles a
    // row, while the streaming kernel's 5 cycles cost a CTA with 200 KB of shared memory for every 32 dimensions.
    constexpr size_t SMALL_NODE = 2048;
    // The host does not know how many nodes a level has: it launches for the most there can be, and asks from here on, where
    // that bound would get out of hand.
    constexpr size_t ASK_LEVEL = 12;
    Pool pool{dev, {}};
    NodeInfo *nodes = pool.get<NodeInfo>(cap_nodes);
    uint32_t *perm = pool.get<uint32_t>(n), *perm2 = pool.get<uint32_t>(n), *keys = pool.get<uint32_t>(n);
    LevelInfo *levels = pool.get<LevelInfo>(2);
    int *error = pool.get<int>(1);
    const size_t n_chunks = (n + MEAN_CHUNK - 1) / MEAN_CHUNK;
    float *partial = n > SMALL_NODE ? pool.get<float>((n_chunks + n / SMALL_NODE + 2) * dim) : nullptr, *spread = nullptr;
    ChunkInfo *chunks = nullptr;
    size_t spread_cap = 0, chunk_cap = 0;
    auto room_for_chunks = [&](size_t level_nodes) {
        if (n_chunks + level_nodes <= chunk_cap) return;
        chunk_cap = n_chunks + 2 * level_nodes + 1024;
        chunks = pool.get<ChunkInfo>(chunk_cap);
    };
    const bool vec = dim % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0; // rows of whole 16-byte pieces
    const auto spread_kernel = vec ? node_spread_stream_kernel<true> : node_spread_stream_kernel<false>;
    VQB_CUDA_CHECK(cudaFuncSetAttribute(spread_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, NS_SMEM));
    const size_t groups = (dim + 31) / 32;
    float *cent = static_cast<float *>(dev.alloc(sizeof(float) * cap_nodes * dim));
    int32_t *left = static_cast<int32_t *>(dev.alloc(sizeof(int32_t) * cap_nodes)), *right = static_cast<int32_t *>(dev.alloc(sizeof(int32_t) * cap_nodes));
    try {
        dev.zero(error, sizeof(int));
        room_for_chunks(2);
        launch_following(init_tree_kernel, grid_for(n, 256, (unsigned)dev.sm_count() * 8), 256, 0, st, n, max_depth > 0 && n > 1 ? 1 : 0, perm, nodes, chunks, levels);
        dev.count_launch();
        LevelInfo known = {0, 1, 0, 0}; // the last level that the host has asked about
        auto ask = [&](size_t l) {
            int herr = 0;
            dev.download(&herr, error, sizeof(int), &known, levels + (l & 1), sizeof known);
            if (herr == NS_ERR_WAIT) throw Error(100, "tsvq: a wait inside the node statistics kernel ran out");
            if (herr) throw Error(herr, "values are not comparable (NaN in the training data)");
        };
        size_t most = 1; // nodes that the level can have
        for (size_t l = 0;; ++l) {
            const LevelInfo *level = levels + (l & 1);
            if (l >= ASK_LEVEL) {
                ask(l);
                if (known.count == 0) break;
                most = (size_t)known.count;
            }
            const bool deepest = l >= max_depth, small = n / most <= SMALL_NODE;
            if (!deepest && most > spread_cap) {
                spread_cap = 2 * most;
                spread = pool.get<float>(spread_cap * dim);
            }
            if (small) {
                KernelScope ks(dev, "tsvq_node_stats");
                // us a build, a warp / a CTA per node and 32 dimensions from 150 rows on: 100,000 x 128, depth 10 1157 / 1110; 2,475 x 122, depth 9
                // 414 / 324; 20,000 x 64, depth 8 464 / 417.  (From 600 rows on 1097, 339, 422.)
                if (n / most >= 150) {
                    const auto kernel = vec ? node_stats_stream_kernel<true> : node_stats_stream_kernel<false>;
                    VQB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STREAM_SMEM));
                    launch_following(kernel, grid_for(most * groups, 1, 1u << 30), STREAM_THREADS, STREAM_SMEM, st, x, dim, perm, nodes, level, cent, spread);
                } else launch_following(vec ? node_stats_kernel<true> : node_stats_kernel<false>, grid_for(most * groups, WR_WARPS, 1u << 30), 32 * WR_WARPS, 0, st, x, dim, perm, nodes, level, cent, spread);
                dev.count_launch();
            } else {
                {
                    KernelScope ks(dev, "tsvq_node_means");
                    const auto kernel = vec ? chunk_sums_kernel<true> : chunk_sums_kernel<false>;
                    VQB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STREAM_SMEM));
                    launch_following(kernel, grid_for((n_chunks + most) * groups, 1, 1u << 30), STREAM_THREADS, STREAM_SMEM, st, x, dim, perm, level, chunks, partial);
                    launch_following(node_mean_kernel, grid_for(most * dim, 128, 1u << 30), 128, 0, st, nodes, level, dim, partial, cent);
                    dev.count_launch();
                    dev.count_launch();
                }
                if (!deepest) {
                    KernelScope ks(dev, "tsvq_node_spreads");
                    launch_following(spread_kernel, grid_for(most * groups, 1, 1u << 30), NS_THREADS, NS_SMEM, st, x, dim, perm, nodes, level, cent, spread, error);
                    dev.count_launch();
                }
            }
            if (deepest) {
                launch_following(no_children_kernel, grid_for(most, 256, 1u << 30), 256, 0, st, level, left, right);
                dev.count_launch();
                ask(l);
                break;
            }
            {
                KernelScope ks(dev, "tsvq_split");
                cudaLaunchConfig_t cfg = {};
                // CTAs of a node by its rows (on average), us a build: 100,000 x 128, depth 10 1319 with eight above 2048 rows and keys in memory, 1241
                // with keys in shared memory, 1176 like this; 300,000 x 32 2526, 2439, 2283; 2,475 x 122, depth 9 494, 434, 417.  (One up to 16,384,
                // then eight: 1192, 2272, 418.)
                const size_t rows = n / most;
                const unsigned cluster = rows <= 4096 ? 1u : rows <= 8192 ? 2u : rows <= 16384 ? 4u : (unsigned)SP_CLUSTER;
                const size_t split_smem = sizeof(uint32_t) * std::min<size_t>(SP_KEYS, 2 * (rows / cluster + 1)); // (nodes are halves, but for ties)
                VQB_CUDA_CHECK(cudaFuncSetAttribute(split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(sizeof(uint32_t) * SP_KEYS)));
                cfg.gridDim = dim3((unsigned)most * cluster);
                cfg.blockDim = dim3(SP_THREADS);
                cfg.dynamicSmemBytes = split_smem;
                cfg.stream = st;
                cudaLaunchAttribute attr[2] = {};
                attr[0].id = cudaLaunchAttributeClusterDimension;
                attr[0].val.clusterDim.x = cluster;
                attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
                attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization; // like launch_following
                attr[1].val.programmaticStreamSerializationAllowed = 1;
                cfg.attrs = attr;
                cfg.numAttrs = 2;
                VQB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, split_kernel, x, dim, (const uint32_t *)perm, perm2, nodes, level, (const float *)spread, keys, (unsigned)(split_smem / sizeof(uint32_t)), error));
                dev.count_launch();
            }
            room_for_chunks(std::min(2 * most, n));
            launch_following(next_level_kernel, 1, 1024, 0, st, nodes, level, levels + ((l + 1) & 1), l + 1 < max_depth ? 1 : 0, left, right, chunks);
            dev.count_launch();
            std::swap(perm, perm2);
            most = std::min(2 * most, n);
        }
        out.dim = dim;
        out.nodes = (size_t)(known.first + known.count);
        out.h_left.resize(out.nodes);
        out.h_right.resize(out.nodes);
        dev.download(out.h_left.data(), left, sizeof(int32_t) * out.nodes, out.h_right.data(), right, sizeof(int32_t) * out.nodes);
    } catch (...) {
        cudaStreamSynchronize(st);
        dev.release(cent), dev.release(left), dev.release(right);
        throw;
    }
    out.centroids = cent;
    out.left = left;
    out.right = right;
}

constexpr size_t TQ_GROUP_DIM = 256;

template <int METRIC, bool VEC, int NP>
static void launch_group(CudaDevice &dev, const TsvqTree &t, double p, const float *x, size_t n, uint16_t *out_f16, uint32_t *leaf)
{
    tsvq_quantize_group_kernel<METRIC, VEC, NP><<<grid_for(n, 32, (unsigned)dev.sm_count() * 16), 256, 0, dev.stream()>>>(x, n, (int)t.dim, t.centroids, t.left, t.right,
                                                                                                                    (float)p, out_f16, leaf);
    VQB_CUDA_CHECK(cudaGetLastError());
    dev.count_launch();
}

template <int METRIC, bool VEC>
static void launch_group(CudaDevice &dev, const TsvqTree &t, double p, const float *x, size_t n, uint16_t *out_f16, uint32_t *leaf)
{
    if (t.dim <= 32) launch_group<METRIC, VEC, 1>(dev, t, p, x, n, out_f16, leaf);
    else if (t.dim <= 64) launch_group<METRIC, VEC, 2>(dev, t, p, x, n, out_f16, leaf);
    else if (t.dim <= 128) launch_group<METRIC, VEC, 4>(dev, t, p, x, n, out_f16, leaf);
    else launch_group<METRIC, VEC, 8>(dev, t, p, x, n, out_f16, leaf);
}

template <int METRIC>
static void launch_quantize(CudaDevice &dev, const TsvqTree &t, double p, const float *x, size_t n, uint16_t *out_f16, uint32_t *leaf)
{
    KernelScope ks(dev, "tsvq_quantize");
    if constexpr (METRIC == M_SQ || METRIC == M_EUCLID) {
        if (t.dim <= TQ_GROUP_DIM && getenv("VQB_TSVQ_SERIAL_WALK") == nullptr) {
            const bool vec = t.dim % 4 == 0 && reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(out_f16) % 8 == 0;
            if (vec) launch_group<METRIC, true>(dev, t, p, x, n, out_f16, leaf);
            else launch_group<METRIC, false>(dev, t, p, x, n, out_f16, leaf);
            return;
        }
    }
    const size_t tile_smem = sizeof(float) * TQ_ROWS * (t.dim + 4);
    const bool aligned = reinterpret_cast<uintptr_t>(x) % 16 == 0 && reinterpret_cast<uintptr_t>(out_f16) % 16 == 0;
    if (t.dim % 8 == 0 && tile_smem <= 200 * 1024 && aligned && getenv("VQB_TSVQ_SERIAL_WALK") == nullptr) {
        allow_shared_memory(dev, tsvq_quantize_tile_kernel<METRIC>);
        const size_t tiles = (n + TQ_ROWS - 1) / TQ_ROWS;
        const unsigned per_sm = (unsigned)std::max<size_t>(1, std::min<size_t>(8, (220 * 1024) / (tile_smem + 1024)));
        const unsigned grid = (unsigned)std::min<size_t>(tiles, (size_t)dev.sm_count() * per_sm);
        tsvq_quantize_tile_kernel<METRIC><<<grid, TQ_ROWS, tile_smem, dev.stream()>>>(x, n, (int)t.dim, t.centroids, t.left, t.right, (float)p, out_f16, leaf);
        VQB_CUDA_CHECK(cudaGetLastError());
        dev.count_launch();
        return;
    }
    tsvq_quantize_kernel<METRIC><<<grid_for(n, 128, (unsigned)dev.sm_count() * 16), 128, 0, dev.stream()>>>(x, n, t.dim, t.centroids, t.left, t.right, (float)p,
                                                                                                     out_f16, leaf);
    VQB_CUDA_CHECK(cudaGetLastError());
    dev.count_launch();
}

void tsvq_quantize(CudaDevice &dev, const TsvqTree &t, int metric, double p, const float *x, size_t n, uint16_t *out_f16, uint32_t *leaf)
{
    if (n == 0) return;
    switch (metric) {
    case M_SQ: launch_quantize<M_SQ>(dev, t, p, x, n, out_f16, leaf); break;
    case M_EUCLID: launch_quantize<M_EUCLID>(dev, t, p, x, n, out_f16, leaf); break;
    case M_COSINE: launch_quantize<M_COSINE>(dev, t, p, x, n, out_f16, leaf); break;
    case M_MANHATTAN: launch_quantize<M_MANHATTAN>(dev, t, p, x, n, out_f16, leaf); break;
    case M_CHEBYSHEV: launch_quantize<M_CHEBYSHEV>(dev, t, p, x, n, out_f16, leaf); break;
    case M_MINKOWSKI: launch_quantize<M_MINKOWSKI>(dev, t, p, x, n, out_f16, leaf); break;
    case M_HAMMING: launch_quantize<M_HAMMING>(dev, t, p, x, n, out_f16, leaf); break;
    default: throw Error(90, "unknown metric");
    }
}

void tsvq_release(CudaDevice &dev, TsvqTree &t)
{
    dev.release(t.centroids), dev.release(t.left), dev.release(t.right);
    t.centroids = nullptr, t.left = nullptr, t.right = nullptr;
}

} // namespace vqb
