// pq_tc.cu -- product-quantizer nearest-centroid search (sub-spaces of 4 or 8 values) with the scores on the tensor cores.
//
// Replaces the per-point scan of src/utils.rs:59-73 (training) and src/pq.rs:159-182 (encode) for the Euclidean metrics and,
// when encoding, cosine.
//
// Scores.  S_j = |c_j|^2/2 - x.c_j ranks the centroids like the squared distance (|x - c_j|^2 = |x|^2 + 2 S_j), for x and c
// taken relative to any common point mu (the mean of the sub-space's centroids here).  Both operands are split into two
// binary16 numbers, x = xh + xl and c = ch + cl, after scaling by powers of two that keep them in range, and tcgen05.mma
// accumulates xh.(-ch) + xh.(-cl) + xl.(-ch) + the half norm (two parts) in f32 in tensor memory: half the MMAs of a split into TF32
// numbers (K = 16 instead of 8 per step at the same cycles).
//
// Fixed point.  What a row needs is the index of its smallest score and whether a second one is close.  The last step of the
// chain adds 2^23 and a row constant K0, and the row's operand carries a factor sigma such that
//     T_j = sigma S_j + K0   lies in [8, 65400]   for every centroid (Cauchy-Schwarz: -min(|x|^2/2, |x| rho) <= S_j <= |x| rho + rho^2/2).
// 2^23 + T_j has T_j, rounded to an integer, in the low 16 bits of its f32 representation: tcgen05.ld.pack::16b delivers two of
// them per register and one 3-input packed minimum (2 cycles of the integer pipe, like the f32 one) looks at four values
// instead of two.  The minimum of every score, which bounded this kernel, costs half, and so does reading tensor memory.
//
// Decision.  Minima of the 16 blocks of 16 consecutive columns and of the 16 classes of columns equal modulo 16, even and odd
// columns side by side in a register.  Two columns differ in their block or in their class, so exactly one T_j lies within M of
// the smallest <=> exactly one block minimum and exactly one class minimum do, and they give its column.  Everything else
// (close scores, ties, NaN / infinity) is put into a queue of the warp in shared memory, with the set of blocks and classes that
// came close; every 32 entries the warp evaluates those columns with the reference's own f32 arithmetic, one entry per lane
// (strict '<' in ascending index, sqrt inside the comparison for the Euclidean metric).  The result equals the exact scan's bit
// for bit.
//
// Bound behind M.  In units of T (sigma (|x|^2 + rho^2) <= 65300, which covers sigma (|x| + rho)^2 / 2):
//   last step: the tensor core aligns its addends to 2^23 and cuts each towards zero two bits below the unit (measured: 1, 2, 8 and
//   16 fractional addends beside 2^23 give errors of 0.25 per addend and one unit downwards for the result).  2^23, K0 and the
//   padding are whole numbers, so that only the accumulator of the steps before is cut: error in (-1.25, 0.25).  How it cuts is not
//   documented, so tests/test_gpu_pq_fixed_point.py measures T against f64: -1.02 .. 0.27 in all, over both widths, cosine, offsets, far
//   and tight centroids
//   steps before: partial sums up to 2^16 in f32: 0.02 each; dropped xl.cl: sd * 8 * 4 * 2^-12 = 0.06, the low parts' rounding as much
//   again; half norm in f32 9u and in two parts 2^-24: 0.04; x - mu and c - mu, u each: 0.01
//   the reference's own arithmetic prefers w over a only if D_w <= D_a (1 + 4u) with (sd + 2)u each: 24u * 65300 = 0.1
//   => T_w <= T_best + 1.5 + 2 * 0.17 + 0.1, i.e. a difference of at most 1.  M = 3 leaves room for twice what was measured.
//
// Far centroids.  One centroid far from the others would stretch the range for all.  Those farther from mu than four times the
// mean distance (mu: the mean of the rest, found in up to six rounds) are left out: rho covers the others.  The producers leave a
// lower bound of what a far one can score against the row, lim^2/2 - lim |x|, in shared memory; a row that has it within reach is
// queued and looks at the far ones as well.  Columns beyond k, far ones and those that are not finite hold T = 57344; a smallest
// value up there is decided by a scan of all centroids.  Rows that are not finite, too far or too large for f32 get an operand of
// zeros: all columns tie, everything is scanned.  So does a sub-space whose
// radius leaves f32; with a NaN in centroid 0, where the reference's scan starts, the answer is 0 without one.
// (500,000 x 128, m 16, k 256, encode, before -> now: rows of normal values 358 -> 260 us; 64 clusters of standard deviation 0.05 / 0.001
// and distance 1: 666 -> 480 / 6100 -> 1640 us; values around 100: 6400 -> 255 us, which the uncentred scores could not separate.  Ties,
// 300,000 x 128: rows on centroids 212 -> 144, each centroid twice 3750 -> 254, four distinct centroids 3750 -> 1665, all equal 3745 -> 2520,
// rows and centroids of 0 and 1 2605 -> 1350 us.)
//
// Cosine (src/distances.rs:141-150).  1 - x.c / (|x| |c|) ranks like S_j = -x.(c_j / |c_j|), with the norm that the reference
// computes and a zero vector for a zero norm (its distance is 1, like a score of 0): no half norms, mu = 0, rho = 1.  The
// reference's quotient carries (2d + 6)u and its difference from 1 another 2u: 48u |x|, 0.1 units of T.  Norms outside
// [1e-17, 1e18] (products that underflow or overflow) void the row, or the sub-space if it is a centroid's.
//
// CTA (1 per SM, persistent, 896 threads), owning up to 4 consecutive sub-spaces (groups share the row tiles).  A unit is one
// 128-row tile of one sub-space; it uses one of the two 128 x 256 f32 accumulators, in two halves of 128 columns.
//   warps 0-3    MMA issuers, one per accumulator half; warp 0 first loads the group's operand-B tiles (TMA, no multicast), warp 1
//                owns tensor memory
//   warps 4-11   take the row tile that TMA has brought into shared memory (two buffers), scale and split the slices (two sub-spaces a
//                warp) and write operand-A tiles, one stage per sub-space
//   warps 12-27  epilogue: a team of four warps per sub-space (one row per lane, one TMEM lane quadrant per warp)
// Every wait is bounded; on expiry the CTA records a code, stops issuing, frees tensor memory and the host raises an error.
//
// Measured, 1M x 128, m 16, k 256: a training pass 0.643 (0.613 and 0.030 for the pairs left to an exact kernel) -> 0.38 ms, an
// encode to f16 rows 0.682 -> 0.43 ms (with 32-bit codes too 0.696 -> 0.470), against f32 scores of split-TF32 operands with one f32
// minimum each.  Per unit 880 cycles; the parts alone: hand-over of the barriers 500, with the producers 720, with the epilogue 860; the
// MMAs take 385, the minima 256 of a scheduler's integer pipe.  What each choice brought (ms a pass, the others as they are):
//   * one issuer per accumulator half instead of one per accumulator (0.46), and those instead of one in all (0.71): a half is idle
//     from its release until its issuer has seen it, and an issuer that waits for one half keeps the other waiting
//   * eight producer warps instead of four (0.48): 150 dependent instructions a slice, 5 cycles each, are what a warp takes
//   * four teams of four warps with 72 registers, whose loads wait for the first half's minima, instead of three with 96 that load a
//     half at once (0.49): more warps in flight count for more than the time a half stays occupied
//   * rows by TMA, and 64- and 32-byte operand rows, which make room for them: loaded by the producers' lanes, 32 rows an
//     instruction, they keep the L1 cache busy for 256 cycles a unit (0.40)
//   * an encode leaves one byte per pair; pq_expand_kernel turns them into rows and 32-bit codes with whole-line stores, 0.06 ms
//     (16-byte pieces stored from here: 0.49 in all)
// The constant in a step of its own (K = 48) rather than beside the last products (K = 32): eleven cut addends instead of one need M = 7, with
// 0.6 units to spare for how the tensor core cuts instead of 1.1, and queue up to twice the rows.  Uniform rows are 5 to 7 % faster with two steps
// (1M x 128, m 16, k 256 at the power limit: encode 469 / 442 us, fit of 10 iterations 5,300 / 4,960), clustered ones slower (500,000 rows in 64
// clusters, standard deviation 0.05 of their distance: 443 / 589, 4,890 / 6,010; 0.1: 321 / 378, 3,750 / 4,210).  Rows that each producer warp fetches
// for itself instead of one copy for all eight gained nothing with three steps (1M 466.7 / 466.0) and cost short calls 4 % (cosine, 60,001 x 96, k 200:
// 36.7 / 35.1).
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "assign_reg.cuh"
#include "cuda_device.hpp"
#include "pq_tc.hpp"
#include "tma_host.hpp"
#include "umma.cuh"

namespace vqb {

namespace {

constexpr int BM = (int)PQ_TC_TILE, BN = 256, MAXM = 64, NTHREADS = 32 * (4 + 8 + 16);
constexpr int QCAP = 64; // queue entries per epilogue warp: fewer than 32 wait, at most 32 are added at a time
constexpr float COS_MIN = 1e-17f, COS_MAX = 1e18f;  // cosine: norms that the scores can be trusted for
constexpr float RHO_MIN = 1e-14f, RHO_MAX = 1e15f;  // Euclidean: radii for which neither 2^+-96 scalings nor distances leave f32
constexpr float SQ_MAX = 5e36f;               // rows beyond: the reference's own distances could overflow
constexpr float T_RANGE = 65300.0f;
constexpr float CR_MIN = 6.2e-5f;             // below: no longer a normal binary16 number
constexpr float SPLIT = 1.5f * 134217728.0f;  // 1.5 2^27: adding it rounds to a multiple of 16
constexpr uint32_t T_HIGH = 57344u - 16u;     // the padding columns' T, less the window

// per-sub-space constants (32 floats): -mu[16], then
constexpr int SUB_RHO2 = 16, SUB_SCALE = 17, SUB_SCALE2 = 18, SUB_FLAGS = 19, SUB_LIM = 20, SUB_MASK = 24, SUB_FLOATS = 32;
constexpr uint32_t SUB_VOID = 1u, SUB_FAR = 2u, SUB_NAN0 = 4u; // NAN0: every distance to centroid 0 is NaN, where the scan starts and stays

// scratch layout (floats)
constexpr size_t OFF_B1 = 0;                                      // [MAXM][256] rows of 32 halves: operand B, K slots 0 .. 31
constexpr size_t OFF_B2 = OFF_B1 + (size_t)MAXM * BN * 16;        // [MAXM][256] rows of 16 halves: K slots 32 .. 47
constexpr size_t OFF_C16 = OFF_B2 + (size_t)MAXM * BN * 8;        // [MAXM][256] rows of up to 8 halves
constexpr size_t OFF_SUB = OFF_C16 + (size_t)MAXM * BN * 4;       // [MAXM][32]
constexpr size_t OFF_STATS = OFF_SUB + (size_t)MAXM * SUB_FLOATS; // 2 x u64: pairs that went through the queues, unused
constexpr size_t SCRATCH_FLOATS = OFF_STATS + 4;

// How the chain's K slots (16 per MMA) are used for each width.  Slots 0 .. 31 lie in a tile of 64-byte rows (64B swizzle), the rest
// in one of 32-byte rows (32B swizzle): 128-byte rows would leave no room for the row tiles.
template <int SD> struct Slots;
template <> struct Slots<4> {
    static constexpr int STEPS = 2, NORM = 12, CONST = 16, M = 3;
};
template <> struct Slots<8> {
    static constexpr int STEPS = 3, NORM = 24, CONST = 32, M = 3;
};
template <int SD> constexpr uint32_t A1_BYTES = BM * 64;                            // a stage
template <int SD> constexpr uint32_t A2_BYTES = Slots<SD>::STEPS == 3 ? BM * 32 : 0;
template <int SD> constexpr uint32_t A_BYTES = A1_BYTES<SD> + A2_BYTES<SD>;
template <int SD> constexpr uint32_t B1_BYTES = BN * 64;                            // a sub-space
template <int SD> constexpr uint32_t B2_BYTES = Slots<SD>::STEPS == 3 ? BN * 32 : 0;
template <int SD> constexpr uint32_t B_BYTES = B1_BYTES<SD> + B2_BYTES<SD>;
template <int SD> constexpr uint32_t RAW_BYTES = BM * 4 * SD * 4;                   // a row tile

struct alignas(8) PqBarriers {
    unsigned long long afull[4], aempty[4], bfull, rfull[2], rempty[2]; // a...: per sub-space; r...: per row-tile buffer
    unsigned long long tfull[8], tempty[8];                             // [2 ss + half]
    uint32_t tmem_base;
    int abort_flag;
};

struct PqTcParams {
    AssignParams a;
    const float *sub; // [m][32]
    unsigned long long *stats;
    int *error;
    float *dbg_scores;              // optional [n][m][256]: scores, or T with
    float *dbg_frames;              // [n][m][2]: sigma and K0
    uint16_t first[MAXM / 4 + 1];   // CTAs first[g] .. first[g + 1] - 1 serve group g
};

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi)
{
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ uint32_t min_u16x2(uint32_t a, uint32_t b)
{
    uint32_t r;
    asm("min.u16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

__device__ __forceinline__ uint32_t min3_u16x2(uint32_t a, uint32_t b, uint32_t c) { return __vimin3_u16x2(a, b, c); } // one instruction on sm_100

// two f32 numbers in one register pair, and what the FMA pipe does with both at once
using F2 = unsigned long long;
__device__ __forceinline__ F2 pair2(float a, float b)
{
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float lo2(F2 v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float hi2(F2 v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b)
{
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b)
{
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c)
{
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

__device__ __forceinline__ float sqrt_approx(float v)
{
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

template <int SD>
constexpr size_t PQ_TC_SMEM = 1024 + 4 * (size_t)B_BYTES<SD> + 4 * (size_t)A_BYTES<SD> + 2 * (size_t)RAW_BYTES<SD> + 4 * SUB_FLOATS * sizeof(float) +
                              16 * QCAP * sizeof(uint4) + 4 * 4 * BM * sizeof(uint16_t) + sizeof(PqBarriers) + 64;

// What a row contributes besides its (shifted) values: the factor of its operand, the half-norm factor and the two row constants.
struct RowFrame {
    float mul, cr, k0;
    uint32_t far; // no far centroid can have a T below this
    bool ok;
};

// sq = |x - mu|^2
template <bool COSINE> __device__ __forceinline__ RowFrame row_frame(float sq, const float *sub)
{
    RowFrame f;
    const float4 c = *reinterpret_cast<const float4 *>(sub + SUB_RHO2); // rho^2 (rounded up), scale, scale^2, flags
    const uint32_t flags = __float_as_uint(c.w);
    float low, sigma;
    if (COSINE) {
        const float norm = sqrt_approx(sq) * 1.000002f; // not below |x| |unit vector|
        low = norm;
        sigma = __fdividef(T_RANGE, 2.0f * norm);
        f.cr = 0.0f;
        f.mul = 0.5f * sigma;
        f.ok = norm >= COS_MIN && norm <= COS_MAX && !(flags & SUB_VOID);
    } else {
        // eleven significant bits, rounded down: cr is a binary16 number as well
        f.cr = __uint_as_float(__float_as_uint(__fdividef(T_RANGE, (sq * 1.000001f + c.x) * c.z)) & 0xFFFFE000u);
        low = 0.5f * sq;
        sigma = f.cr * c.z;
        f.mul = f.cr * c.y;
        f.ok = sq < SQ_MAX && f.cr >= CR_MIN && !(flags & SUB_VOID);
    }
    // a whole number (1.5 2^23 rounds it), 12 to spare after rounding to binary16
    f.k0 = fmaf(low, sigma * 1.001f, 12582912.0f + 12.0f) - 12582912.0f;
    f.far = 0xFFFFu;
    if (flags & SUB_FAR) {
        const float lim = sub[SUB_LIM], norm = sqrt_approx(sq) * 1.000001f;
        const float t = norm < lim ? (0.5f * lim - norm) * lim * sigma + 0.999f * f.k0 - 16.0f : 0.0f;
        f.far = (uint32_t)fminf(fmaxf(t, 0.0f), 65535.0f);
    }
    return f;
}

// Minima of 64 more columns (two per register): hb = their four blocks of 16, ga = the classes.
template <bool FIRST> __device__ __forceinline__ void fold64(const uint32_t (&v)[32], uint32_t *hb, uint32_t (&ga)[8])
{
#pragma unroll
    for (int t = 0; t < 8; ++t) {
        if (FIRST) {
            ga[t] = min3_u16x2(v[t], v[8 + t], v[16 + t]);
            ga[t] = min_u16x2(ga[t], v[24 + t]);
        } else {
            ga[t] = min3_u16x2(ga[t], v[t], v[8 + t]);
            ga[t] = min3_u16x2(ga[t], v[16 + t], v[24 + t]);
        }
    }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        const uint32_t *w = v + 8 * b;
        hb[b] = min3_u16x2(min3_u16x2(w[0], w[1], w[2]), min3_u16x2(w[3], w[4], w[5]), min_u16x2(w[6], w[7]));
    }
}

// The queued rows of one warp, one per lane, with the reference's arithmetic.  Entry: x = tile, y = row in the tile | classes << 16
// (bit c: columns = c modulo 16 are candidates), z = blocks (bit 2 i + p: block i, columns of parity p), w = Q_WHOLE: all centroids;
// Q_FAR: the far ones as well.  Returns whether this lane's assignment changed.
constexpr uint32_t Q_WHOLE = 1u, Q_FAR = 2u;

template <int SD, bool TRAIN, int METRIC>
__device__ __noinline__ bool pq_queue_drain(const PqTcParams &Q, const uint4 *queue, const float *sub, int count, int s, int lane)
{
    const AssignParams &P = Q.a;
    bool moved = false;
    const bool mine = lane < count;
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    if (mine) e = queue[lane];
    const unsigned long long row = (unsigned long long)e.x * BM + (e.y & 127u);
    float x[SD];
    if (mine) {
        load_slice<SD>(x, P.x + row * P.ld + (size_t)s * SD, true);
    } else {
#pragma unroll
        for (int i = 0; i < SD; ++i) x[i] = 0.0f;
    }
    const float na = METRIC == M_COSINE ? norm_chain(x, SD, 1) : 0.0f;
    const float *cbs = P.centroids + (size_t)s * P.k * SD;
    float bd = VQB_INF;
    int bi = 0x7fffffff;
    bool nan0 = false;
    auto distance = [&](int j) { // (Euclidean: its square)
        float cv[SD];
        load_centroid<SD>(cv, cbs + (size_t)j * SD);
        return METRIC == M_COSINE ? reg_dist<SD, M_COSINE>(x, cv, 0.0f, na, norm_chain(cv, SD, 1)) : reg_dist<SD, M_SQ>(x, cv, 0.0f, 0.0f, 0.0f);
    };
    auto look = [&](int j) {
        float d = distance(j);
        if (METRIC == M_EUCLID) d = __fsqrt_rn(d);
        if (j == 0) nan0 = !(d == d);
        if (d < bd || (d == bd && j < bi)) {
            bd = d;
            bi = j;
        }
    };
    // many candidates (ties): the lanes go through all centroids together, whose loads are then the same for all
    constexpr int U = 4; // distances in flight: each is a chain of additions
    if (P.k < U && (e.w & Q_WHOLE)) e.y |= 0xFFFF0000u, e.z = 3u;
    const bool all = P.k >= U && ((e.w & Q_WHOLE) || __popc(e.z) * __popc(e.y >> 16) >= 256);
    if (__float_as_uint(sub[SUB_FLAGS]) & SUB_NAN0) {
        nan0 = true;
    } else if (__any_sync(0xffffffffu, all)) {
        // in ascending order a centroid that is not below the best one's square cannot have the smaller root: the root is taken of new
        // minima only (300,000 x 128, m 16, k 256, all centroids equal: encode 4.25 -> 2.52 ms with both changes, 4.04 with this one)
        float best = VQB_INF;
        for (int j = 0;;) {
            float d[U];
#pragma unroll
            for (int u = 0; u < U; ++u) d[u] = distance(j + u);
            if (j == 0) nan0 = !(d[0] == d[0]);
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (d[u] < best) {
                    const float r = METRIC == M_EUCLID ? __fsqrt_rn(d[u]) : d[u];
                    if (r < bd) best = d[u], bd = r, bi = j + u;
                }
            if (j + U >= P.k) break;
            j = min(j + U, P.k - U); // (some of the last step's a second time: none of them is below the best)
        }
    }
    if (!all) {
        bd = VQB_INF, bi = 0x7fffffff, nan0 = false;
        uint32_t blocks = e.z;
        while (blocks) {
            const int bit = __ffs(blocks) - 1;
            blocks &= blocks - 1;
            uint32_t c = (e.y >> 16) & ((bit & 1) ? 0xAAAAu : 0x5555u);
            while (c) {
                const int j = (bit >> 1) * 16 + __ffs(c) - 1;
                c &= c - 1;
                if (j < P.k) look(j);
            }
        }
        if (e.w & Q_FAR)
            for (int w = 0; w < BN / 32; ++w) {
                uint32_t far = __float_as_uint(sub[SUB_MASK + w]);
                while (far) {
                    look(w * 32 + __ffs(far) - 1);
                    far &= far - 1;
                }
            }
    }
    if (mine) {
        const int idx = (bi == 0x7fffffff || nan0) ? 0 : bi; // nothing below +inf, or the reference's scan starts at a NaN
        uint8_t *cp = reinterpret_cast<uint8_t *>(P.codes) + row * (unsigned long long)P.m + s;
        if (!TRAIN || *cp != (uint8_t)idx) {
            moved = true;
            *cp = (uint8_t)idx;
        }
    }
    if (lane == 0) atomicAdd(Q.stats, (unsigned long long)count);
    __syncwarp(); // the entries are read: the caller may add new ones
    return moved;
}

// DUMP: diagnostics in place of codes, 1: the chain's result without the fixed-point constants, as scores; 2: T itself and the rows' sigma and K0
template <int SD, bool TRAIN, int METRIC, bool WIDE, int DUMP>
__global__ void __launch_bounds__(NTHREADS, 1)
    pq_tc_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_b1, const __grid_constant__ CUtensorMap map_b2,
                 const __grid_constant__ PqTcParams Q)
{
    constexpr bool COSINE = METRIC == M_COSINE;
    constexpr int halves = WIDE ? 2 : 1; // accumulator halves that hold centroids
    using SL = Slots<SD>;
    extern __shared__ unsigned char smem_raw[];
    const AssignParams &P = Q.a;
    unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *b_smem = base;                                                    // [4] 64-byte rows, then [4] 32-byte rows
    unsigned char *a_smem = base + 4 * (size_t)B_BYTES<SD>;                          // the same
    unsigned char *raw_smem = a_smem + 4 * (size_t)A_BYTES<SD>;                      // [2] row tiles
    float *sub_s = reinterpret_cast<float *>(raw_smem + 2 * (size_t)RAW_BYTES<SD>);  // [4][32]
    uint4 *queues = reinterpret_cast<uint4 *>(sub_s + 4 * SUB_FLOATS);               // [16][QCAP]
    uint16_t *far_s = reinterpret_cast<uint16_t *>(queues + 16 * QCAP);              // [4][4][128] RowFrame::far of four tiles
    PqBarriers *bars = reinterpret_cast<PqBarriers *>(far_s + 4 * 4 * BM);
    volatile int *abort_flag = &bars->abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31; // (the shuffle: uniform by construction)
    const int m = P.m, k = P.k;
    int g = 0;
    while (blockIdx.x >= Q.first[g + 1]) ++g;
    const uint32_t tile0 = blockIdx.x - Q.first[g], tstep = Q.first[g + 1] - Q.first[g];
    const uint32_t n_tiles = (uint32_t)((P.n + BM - 1) / BM);
    const uint32_t last_rows = (uint32_t)(P.n - (unsigned long long)(n_tiles - 1) * BM); // rows of the last tile
    const int here = min(4, m - 4 * g); // sub-spaces of this group

    if (threadIdx.x == 0) {
        for (int s = 0; s < 4; ++s) {
            mbar_init(&bars->afull[s], 4);
            mbar_init(&bars->aempty[s], halves); // one commit per accumulator half
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bars->rfull[b], 1);
            mbar_init(&bars->rempty[b], 8);
        }
        mbar_init(&bars->bfull, 1);
        for (int b = 0; b < 8; ++b) {
            mbar_init(&bars->tfull[b], 1);
            mbar_init(&bars->tempty[b], 4);
        }
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (uint32_t i = threadIdx.x; i < 4 * A_BYTES<SD> / 16; i += NTHREADS) // the slots that no row uses stay zero
        reinterpret_cast<uint4 *>(a_smem)[i] = make_uint4(0u, 0u, 0u, 0u);
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    after_previous_kernel();
    next_kernel_may_start();
    uint32_t act = 0; // bit ss: sub-space ss of the group takes part (identical in every thread)
#pragma unroll
    for (int ss = 0; ss < 4; ++ss)
        if (ss < here && !(TRAIN && P.active && P.active[g * 4 + ss] == 0)) act |= 1u << ss;
    if (threadIdx.x < here * SUB_FLOATS) sub_s[threadIdx.x] = Q.sub[(size_t)g * 4 * SUB_FLOATS + threadIdx.x];
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = bars->tmem_base;

    if (warp < 4) {
        // ------------------------------------------------ operand B: the group's sub-spaces, once
        const bool leader = elect_one();
        if (warp == 0 && leader && act) {
            mbar_expect_tx(&bars->bfull, (uint32_t)here * B_BYTES<SD>);
            for (int ss = 0; ss < here; ++ss) {
                tma_load_2d(b_smem + (size_t)ss * B1_BYTES<SD>, &map_b1, 0, (g * 4 + ss) * BN, &bars->bfull);
                if (B2_BYTES<SD>) tma_load_2d(b_smem + 4 * (size_t)B1_BYTES<SD> + (size_t)ss * B2_BYTES<SD>, &map_b2, 0, (g * 4 + ss) * BN, &bars->bfull);
            }
        }
        __syncwarp();
        // ------------------------------------------------ MMA issuer of half warp % 2 of accumulator warp / 2: the whole warp walks the loop,
        // so that what it works out is uniform, and one lane issues
        const int acc = warp >> 1, half = warp & 1;
        const uint32_t mine = half < halves ? act >> (2 * acc) & 3u : 0u;
        if (mine) {
            bool ok = mbar_wait(&bars->bfull, 0, abort_flag, Q.error, 12);
            const uint32_t a1 = (smem_u32(a_smem) + 2 * acc * A1_BYTES<SD>) >> 4, a2 = (smem_u32(a_smem) + 4 * A1_BYTES<SD> + 2 * acc * A2_BYTES<SD>) >> 4;
            const uint32_t b1 = (smem_u32(b_smem) + 2 * acc * B1_BYTES<SD> + half * (B1_BYTES<SD> / 2)) >> 4;
            const uint32_t b2 = (smem_u32(b_smem) + 4 * B1_BYTES<SD> + 2 * acc * B2_BYTES<SD> + half * (B2_BYTES<SD> / 2)) >> 4;
            const uint32_t td = tmem_base + acc * BN + half * 128;
            uint32_t phase = 0; // parity of the tile's phases
            for (uint32_t tile = tile0; ok && tile < n_tiles; tile += tstep, phase ^= 1u) { // (after an abort the next wait fails)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    if (!(mine >> h & 1u) || !ok) continue;
                    const int ss = 2 * acc + h;
                    // the columns' last user: the other sub-space if it takes part (in this tile for h = 1), else this one in the tile before
                    const int before = mine == 3u ? ss ^ 1 : ss;
                    const uint32_t parity = (h == 1 && mine == 3u) ? phase : phase ^ 1u;
                    if (!mbar_wait(&bars->afull[ss], phase, abort_flag, Q.error, 14) || !mbar_wait(&bars->tempty[2 * before + half], parity, abort_flag, Q.error, 13)) {
                        ok = false;
                        continue;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    if (leader) {
                        const uint32_t o = (uint32_t)h; // 16 halves = 32 bytes = 2 descriptor units per step
                        umma_f16_n128(td, smem_desc_sw64_at(a1 + o * (A1_BYTES<SD> >> 4)), smem_desc_sw64_at(b1 + o * (B1_BYTES<SD> >> 4)), 0u);
                        umma_f16_n128(td, smem_desc_sw64_at(a1 + o * (A1_BYTES<SD> >> 4) + 2), smem_desc_sw64_at(b1 + o * (B1_BYTES<SD> >> 4) + 2), 1u);
                        if (SL::STEPS == 3) umma_f16_n128(td, smem_desc_sw32_at(a2 + o * (A2_BYTES<SD> >> 4)), smem_desc_sw32_at(b2 + o * (B2_BYTES<SD> >> 4)), 1u);
                        umma_commit(&bars->tfull[2 * ss + half]);
                        umma_commit(&bars->aempty[ss]);
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < 12) {
        // ------------------------------------------------ operand A: scaled and split row slices
        const int r = (warp & 3) * 32 + lane; // row of the tile
        const int pair = (warp - 4) >> 2;     // this warp's sub-spaces: 2 pair, 2 pair + 1
        auto load_tile = [&](uint32_t tile, uint32_t buf) { // rows and columns beyond the matrix arrive as zeros
            mbar_expect_tx(&bars->rfull[buf], RAW_BYTES<SD>);
            tma_load_2d(raw_smem + buf * RAW_BYTES<SD>, &map_x, g * 4 * SD, (int)(tile * BM), &bars->rfull[buf]);
        };
        if (warp == 4 && lane == 0 && act) {
            if (tile0 < n_tiles) load_tile(tile0, 0);
            if (tile0 + tstep < n_tiles) load_tile(tile0 + tstep, 1);
        }
        __syncwarp();
        uint32_t step = 0, buf = 0, rphase = 0; // tiles so far (parity: that of the stages); row-tile buffer and its parity
        bool ok = true;
        for (uint32_t tile = tile0; act && ok && tile < n_tiles; tile += tstep, ++step) {
            if (!mbar_wait(&bars->rfull[buf], rphase, abort_flag, Q.error, 10)) break;
            const unsigned char *raw = raw_smem + buf * RAW_BYTES<SD> + r * (16 * SD);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int ss = 2 * pair + h;
                if (!(act >> ss & 1u) || !ok) continue;
                const float *sub = sub_s + ss * SUB_FLOATS;
                // two values per instruction where the FMA pipe has one (add, fma .f32x2)
                F2 y[SD / 2];
#pragma unroll
                for (int c = 0; c < SD / 4; ++c) {
                    const int chunk = ss * (SD / 4) + c;
                    const ulonglong2 v = *reinterpret_cast<const ulonglong2 *>(raw + ((SD == 8 ? chunk ^ (r & 7) : chunk ^ ((r >> 1) & 3)) << 4));
                    y[2 * c] = v.x, y[2 * c + 1] = v.y;
                    if (!COSINE) {
                        const ulonglong2 mu = reinterpret_cast<const ulonglong2 *>(sub)[c]; // the mean with its sign changed
                        y[2 * c] = add2(y[2 * c], mu.x), y[2 * c + 1] = add2(y[2 * c + 1], mu.y);
                    }
                }
                F2 sq2 = mul2(y[0], y[0]);
#pragma unroll
                for (int i = 1; i < SD / 2; ++i) sq2 = fma2(y[i], y[i], sq2);
                const RowFrame f = row_frame<COSINE>(lo2(sq2) + hi2(sq2), sub);
                uint32_t hi[SD / 2], lo[SD / 2], cc, k0;
                const F2 mul = pair2(f.mul, f.mul), up = pair2(SPLIT, SPLIT), down = pair2(-SPLIT, -SPLIT);
#pragma unroll
                for (int i = 0; i < SD / 2; ++i) {
                    // |y mul| < 2^15: the multiple of 16 next to it and the rest (at most 8) are both binary16 numbers, the rest to 2^-9
                    const F2 head = add2(fma2(y[i], mul, up), down);
                    hi[i] = pack_f16(lo2(head), hi2(head));
                    lo[i] = pack_f16(fmaf(lo2(y[i]), f.mul, -lo2(head)), fmaf(hi2(y[i]), f.mul, -hi2(head)));
                }
                cc = pack_f16(f.cr, f.cr);
                k0 = DUMP == 1 ? 0u : pack_f16(2048.0f, f.k0);
                if (__any_sync(0xffffffffu, !f.ok)) { // (rarely: a vote instead of a select per word)
#pragma unroll
                    for (int i = 0; i < SD / 2; ++i) hi[i] = f.ok ? hi[i] : 0u, lo[i] = f.ok ? lo[i] : 0u;
                    cc = f.ok ? cc : 0u, k0 = f.ok ? k0 : 0u;
                }
                if (DUMP == 2 && tile * (unsigned long long)BM + r < P.n) {
                    float *o = Q.dbg_frames + ((tile * (unsigned long long)BM + r) * m + g * 4 + ss) * 2;
                    o[0] = f.ok ? f.mul * sub[SUB_SCALE] : 0.0f;
                    o[1] = __half2float(__float2half_rn(f.k0));
                }
                if (!mbar_wait(&bars->aempty[ss], (step & 1u) ^ 1u, abort_flag, Q.error, 11)) {
                    ok = false;
                    continue;
                }
                unsigned char *row1 = a_smem + (size_t)ss * A1_BYTES<SD> + (size_t)r * 64;
                const int s1 = (r >> 1) & 3;
                if (SD == 4) {
                    *reinterpret_cast<uint4 *>(row1 + ((0 ^ s1) << 4)) = make_uint4(hi[0], hi[1], hi[0], hi[1]);
                    *reinterpret_cast<uint4 *>(row1 + ((1 ^ s1) << 4)) = make_uint4(lo[0], lo[1], cc, 0u);
                    *reinterpret_cast<uint4 *>(row1 + ((2 ^ s1) << 4)) = make_uint4(k0, 0u, 0u, 0u);
                } else {
                    const uint4 h4 = make_uint4(hi[0], hi[1], hi[2 % (SD / 2)], hi[3 % (SD / 2)]);
                    *reinterpret_cast<uint4 *>(row1 + ((0 ^ s1) << 4)) = h4;
                    *reinterpret_cast<uint4 *>(row1 + ((1 ^ s1) << 4)) = h4;
                    *reinterpret_cast<uint4 *>(row1 + ((2 ^ s1) << 4)) = make_uint4(lo[0], lo[1], lo[2 % (SD / 2)], lo[3 % (SD / 2)]);
                    *reinterpret_cast<uint4 *>(row1 + ((3 ^ s1) << 4)) = make_uint4(cc, 0u, 0u, 0u);
                    unsigned char *row2 = a_smem + 4 * (size_t)A1_BYTES<SD> + (size_t)ss * A2_BYTES<SD> + (size_t)r * 32;
                    *reinterpret_cast<uint4 *>(row2 + (((r >> 2) & 1) << 4)) = make_uint4(k0, 0u, 0u, 0u);
                }
                if (__float_as_uint(sub[SUB_FLAGS]) & SUB_FAR) far_s[(ss * 4 + (step & 3u)) * BM + r] = (uint16_t)f.far;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic writes -> visible to the MMA's reads
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->afull[ss]);
            }
            if (!ok) break;
            // the row tile is used up: once all eight warps say so, its buffer takes the tile after the next
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->rempty[buf]);
            if (warp == 4 && tile + 2 * tstep < n_tiles) {
                ok = mbar_wait(&bars->rempty[buf], rphase, abort_flag, Q.error, 17);
                if (ok && lane == 0) load_tile(tile + 2 * tstep, buf);
                __syncwarp();
            }
            buf ^= 1u;
            if (buf == 0) rphase ^= 1u;
        }
    } else {
        // ------------------------------------------------ epilogue: team (warp - 12) / 4 serves that sub-space of the group
        const int q = warp & 3; // TMEM lane quadrant
        const int ss = (warp - 12) >> 2, s = g * 4 + ss;
        const uint32_t taddr = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(ss >> 1) * BN;
        const float *sub = sub_s + ss * SUB_FLOATS;
        uint4 *queue = queues + (warp - 12) * QCAP;
        const bool any_far = (__float_as_uint(sub[SUB_FLAGS]) & SUB_FAR) != 0;
        uint32_t waiting = 0; // entries in the queue
        bool moved = false;
        const bool on = act >> ss & 1u;
        const uint32_t r = 32u * q + lane;
        const uint32_t n_steps = tile0 < n_tiles ? (n_tiles - tile0 + tstep - 1) / tstep : 0u; // tiles of this CTA
        const bool in_last = r < (tile0 + (n_steps - 1) * tstep == n_tiles - 1 ? last_rows : (uint32_t)BM);
        auto there = [&](uint32_t t) { return t + 1 < n_steps || (t < n_steps && in_last); };
        uint8_t *code = reinterpret_cast<uint8_t *>(P.codes) + ((unsigned long long)tile0 * BM + r) * m + s; // this lane's row of the tile
        const uint32_t code_step = tstep * BM * (uint32_t)m;
        // the previous code of a row is requested while the tile before it is decided: a trip to memory is longer than a unit
        uint32_t next_old = 0;
        if (TRAIN && on && there(0)) next_old = *code;
        for (uint32_t step = 0; on && step < n_steps; ++step, code += code_step) {
            const bool valid = there(step);
            const uint32_t old = next_old;
            if (TRAIN && there(step + 1)) next_old = code[code_step];
            uint32_t hb[16], ga[8];
            bool ok = true;
#pragma unroll
            for (int half = 0; half < halves; ++half) {
                if (!ok) continue;
                if (!mbar_wait(&bars->tfull[2 * ss + half], step & 1u, abort_flag, Q.error, 15)) {
                    ok = false;
                    continue;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint32_t v[32];
                if (DUMP) {
                    const unsigned long long row = (unsigned long long)(tile0 + step * tstep) * BM + r;
                    float x[SD], sq[2] = {0.0f, 0.0f}, shift = 0.0f;
#pragma unroll
                    for (int i = 0; i < SD; ++i) x[i] = 0.0f;
                    if (valid) load_slice<SD>(x, P.x + row * P.ld + (size_t)s * SD, true);
#pragma unroll
                    for (int i = 0; i < SD; ++i) {
                        const float mu = -sub[i], y = x[i] - mu;
                        sq[i & 1] = fmaf(y, y, sq[i & 1]); // (in the producers' order: cr is cut to eleven bits)
                        shift = fmaf(mu, x[i] - 0.5f * mu, shift); // S = S' - y.mu - |mu|^2 / 2
                    }
                    const RowFrame f = row_frame<COSINE>(sq[0] + sq[1], sub);
                    const float sigma = f.cr * sub[SUB_SCALE2];
                    for (int c = 0; c < 4; ++c) {
                        tmem_ld32_issue(taddr + half * 128 + c * 32, v);
                        tmem_wait();
                        if (valid) {
                            float *o = Q.dbg_scores + ((size_t)row * m + s) * BN + half * 128 + c * 32;
#pragma unroll
                            for (int t = 0; t < 32; ++t) {
                                if (DUMP == 2) o[t] = __uint_as_float(v[t]) - 8388608.0f;
                                else o[t] = half * 128 + c * 32 + t < k ? __uint_as_float(v[t]) / sigma - shift : 1e30f;
                            }
                        }
                    }
                } else {
                    tmem_ld32_pack16_issue(taddr + half * 128, v);
                    tmem_wait();
                    if (half == 0) fold64<true>(v, hb, ga);
                    else fold64<false>(v, hb + 8, ga);
                    tmem_ld32_pack16_issue(taddr + half * 128 + 64, v);
                    tmem_wait();
                }
                // the half is in registers: its columns may be overwritten
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->tempty[2 * ss + half]);
                if (!DUMP) fold64<false>(v, hb + 8 * half + 4, ga);
            }
            if (!ok) break;
            if (DUMP) continue;

            uint32_t best2 = 0xFFFFFFFFu;
            {
                constexpr int NB = 8 * halves;
                uint32_t b[NB / 3 + 1];
#pragma unroll
                for (int i = 0; i < NB / 3; ++i) b[i] = min3_u16x2(hb[3 * i], hb[3 * i + 1], hb[3 * i + 2]);
                if (WIDE) best2 = min_u16x2(min3_u16x2(b[0], b[1], b[2]), min3_u16x2(b[3], b[NB / 3 - 1], hb[NB - 1]));
                else best2 = min_u16x2(min3_u16x2(b[0], b[1], hb[6]), hb[7]);
            }
            const uint32_t best = min(best2 & 0xFFFFu, best2 >> 16);
            const uint32_t minus = ((0u - best) & 0xFFFFu) * 0x10001u; // adding it: the distance from the best, never negative
            constexpr uint32_t MM = SL::M * 0x10001u;
            // Sums of weight * min(distance, M) over the blocks (weight W0 + block) and over the classes (W0 + class), both halves of a word
            // at once.  What they lack of M times all weights is the sum of weight * (M - distance) over those within M: one with distance 0
            // gives M weights, two or more at least W0 (M + 1) > M (W0 + 15).
            constexpr uint32_t W0 = 16 * SL::M, NBLK = 8 * halves;
            constexpr uint32_t WB = 2 * SL::M * (NBLK * W0 + NBLK * (NBLK - 1) / 2), WA = SL::M * (16 * W0 + 120);
            uint32_t sb = 0, sb1 = 0, sa = 0, sa1 = 0;
#pragma unroll
            for (uint32_t i = 0; i < NBLK; i += 2) {
                sb = __dp2a_lo(__viaddmin_u16x2(hb[i], minus, MM), (W0 + i) * 0x101u, sb);
                sb1 = __dp2a_lo(__viaddmin_u16x2(hb[i + 1], minus, MM), (W0 + i + 1) * 0x101u, sb1);
            }
#pragma unroll
            for (uint32_t i = 0; i < 8; i += 2) {
                sa = __dp2a_lo(__viaddmin_u16x2(ga[i], minus, MM), (W0 + 2 * i) + ((W0 + 2 * i + 1) << 8), sa);
                sa1 = __dp2a_lo(__viaddmin_u16x2(ga[i + 1], minus, MM), (W0 + 2 * i + 2) + ((W0 + 2 * i + 3) << 8), sa1);
            }
            const uint32_t lb = WB - sb - sb1, la = WA - sa - sa1;
            const uint32_t idx = ((lb * 16u + la - SL::M * 17u * W0) / SL::M) & 0xFFu; // 16 block + class
            const bool whole = best - 1u >= T_HIGH - 1u; // 0: nothing to tell apart; high up: nothing but columns without a centroid
            bool single = max(lb, la) <= SL::M * (W0 + 15u) && !whole;
            // a far centroid may be as close (the entry is written again four tiles on, which takes this unit's end)
            const bool far = any_far && best + SL::M > far_s[(ss * 4 + (step & 3u)) * BM + r];
            single = single && !far;
            const bool later = valid && !single;
            const uint32_t vote = __ballot_sync(0xffffffffu, later);
            if (vote) {
                // one bit per half of a word: min(distance, M) + (65536 - M) wraps to 0 for M and stays at least 1 otherwise
                constexpr uint32_t LESS = (0x10000u - SL::M) * 0x10001u;
                uint32_t blocks = 0, classes = 0;
#pragma unroll
                for (int c = 0; c < 2 * halves; ++c) { // four words at a time: eight bits, weighted by the bytes of dp2a
                    uint32_t bits = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) bits = __dp2a_lo(__viaddmin_u16x2(__viaddmin_u16x2(hb[4 * c + i], minus, MM), LESS, 0x10001u), 0x201u << (2 * i), bits);
                    blocks |= bits << (8 * c);
                }
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t bits = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i) bits = __dp2a_lo(__viaddmin_u16x2(__viaddmin_u16x2(ga[4 * c + i], minus, MM), LESS, 0x10001u), 0x201u << (2 * i), bits);
                    classes |= bits << (8 * c);
                }
                if (later) queue[waiting + __popc(vote & ((1u << lane) - 1u))] = make_uint4(tile0 + step * tstep, r | (classes << 16), blocks, (whole ? Q_WHOLE : 0u) | (far ? Q_FAR : 0u));
                waiting += __popc(vote);
                __syncwarp();
                if (waiting >= 32) {
                    waiting -= 32;
                    moved |= pq_queue_drain<SD, TRAIN, METRIC>(Q, queue + waiting, sub, 32, s, lane);
                }
            }
            if (valid && single && (!TRAIN || idx != old)) {
                moved = true;
                *code = (uint8_t)idx;
            }
        }
        if (waiting) moved |= pq_queue_drain<SD, TRAIN, METRIC>(Q, queue, sub, (int)waiting, s, lane);
        if (TRAIN && __any_sync(0xffffffffu, moved) && lane == 0) atomicOr(P.changed + s, VQB_MOVED_BITS);
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// The encode's outputs from its one-byte codes (codes [n][m]): thread = one (row, sub-space) pair at a time, neighbours in memory next
// to each other, so that every store covers whole lines.  The images of the centroids (c16 [m][256][SD]) are gathered from shared memory
// when they fit (TABLE): 16 bytes per lane from 32 different lines would take 32 cycles of the L1 cache.
template <int SD, bool TABLE>
__global__ void __launch_bounds__(512) pq_expand_kernel(const uint8_t *codes, unsigned long long pairs, int m, int k, const uint16_t *c16, const float *centroids,
                                                        uint16_t *out_f16, uint32_t *out_codes, float *out_f32)
{
    extern __shared__ __align__(16) uint16_t table[];
    using Piece = typename std::conditional<SD == 4, uint2, uint4>::type; // SD halves
    after_previous_kernel();
    next_kernel_may_start();
    if (TABLE) {
        for (uint32_t i = threadIdx.x; i < (uint32_t)m * BN * SD / 8; i += blockDim.x) reinterpret_cast<uint4 *>(table)[i] = __ldg(reinterpret_cast<const uint4 *>(c16) + i);
        __syncthreads();
    }
    // eight codes are requested before the first is used: with one at a time a thread waits for memory once per pair (85 us for 1M x 16)
    constexpr int U = 8;
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    const uint32_t step = (uint32_t)(stride % (uint32_t)m);
    unsigned long long i0 = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    uint32_t s = (uint32_t)(i0 % (uint32_t)m);
    for (; i0 < pairs; i0 += U * stride) {
        uint32_t idx[U];
#pragma unroll
        for (int u = 0; u < U; ++u) idx[u] = i0 + u * stride < pairs ? __ldcs(codes + i0 + u * stride) : 0u;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const unsigned long long i = i0 + u * stride;
            if (i < pairs) {
                if (out_codes) __stcs(out_codes + i, idx[u]);
                if (out_f16) __stcs(reinterpret_cast<Piece *>(out_f16) + i, reinterpret_cast<const Piece *>(TABLE ? table : c16)[s * BN + idx[u]]);
                if (out_f32) {
#pragma unroll
                    for (int c = 0; c < SD / 4; ++c)
                        reinterpret_cast<float4 *>(out_f32)[i * (SD / 4) + c] = __ldg(reinterpret_cast<const float4 *>(centroids) + ((size_t)s * k + min(idx[u], (uint32_t)k - 1u)) * (SD / 4) + c);
                }
            }
            s += step;
            if (s >= (uint32_t)m) s -= (uint32_t)m;
        }
    }
}

// ------------------------------------------------------------------------------------------------
// Operand B of one sub-space by one block of 256 threads (thread j = centroid j, v its values)
// ------------------------------------------------------------------------------------------------
template <int SD> struct OperandSmem {
    float part[8][SD + 1];
    float part1[8];
};

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Row j of operand B (64 halves, see Slots), the binary16 image that an encode writes (src/pq.rs:176-180) and the sub-space's constants.
template <int SD, bool COSINE>
__device__ __forceinline__ void write_operand(const float (&v)[SD], int s, int k, float *scratch, OperandSmem<SD> &sm)
{
    using SL = Slots<SD>;
    const int j = threadIdx.x, warp = j >> 5, lane = j & 31;
    bool finite = true;
#pragma unroll
    for (int i = 0; i < SD; ++i) finite = finite && fabsf(v[i]) < VQB_INF;
    // A distance to a centroid that is not finite is never below another (src/utils.rs:66): its column is like one beyond k.  But the
    // scan starts at centroid 0, and at a NaN it stays.
    const bool mine = j < k && finite;
    bool nan = false;
#pragma unroll
    for (int i = 0; i < SD; ++i) nan = nan || !(v[i] == v[i]);
    const bool lost = __syncthreads_or(j == 0 && (COSINE ? !finite : nan)) != 0;
    float y[SD], mu[SD], norm = 0.0f, rho = 0.0f, lim = 0.0f, half_norm = 0.0f;
    bool far = false, void_sub = false;
    if (COSINE) {
        const float len = norm_chain(v, SD, 1);
#pragma unroll
        for (int i = 0; i < SD; ++i) {
            mu[i] = 0.0f;
            y[i] = mine && len != 0.0f ? __fdiv_rn(v[i], len) : 0.0f;
        }
        void_sub = lost || __syncthreads_or(mine && !(len == 0.0f || (len >= COS_MIN && len <= COS_MAX))) != 0;
        rho = 1.000001f;
    } else {
        bool in = mine;
#pragma unroll 1
        for (int round = 0;; ++round) { // mu = the mean of those that are not far from it
            const float cnt = warp_sum(in ? 1.0f : 0.0f);
#pragma unroll
            for (int i = 0; i < SD; ++i) {
                const float t = warp_sum(in ? v[i] : 0.0f);
                if (lane == 0) sm.part[warp][i] = t;
            }
            if (lane == 0) sm.part[warp][SD] = cnt;
            __syncthreads();
            float c = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; ++w) c += sm.part[w][SD];
            const float inv = __fdividef(1.0f, c);
            float sq = 0.0f;
#pragma unroll
            for (int i = 0; i < SD; ++i) {
                float t = 0.0f;
#pragma unroll
                for (int w = 0; w < 8; ++w) t += sm.part[w][i];
                mu[i] = t * inv;
                y[i] = mine ? v[i] - mu[i] : 0.0f;
                sq = fmaf(y[i], y[i], sq);
            }
            half_norm = 0.5f * sq;
            norm = sqrt_approx(sq) * 1.000001f;
            const float t = warp_sum(in ? norm : 0.0f);
            if (lane == 0) sm.part1[warp] = t;
            __syncthreads();
            float sum = 0.0f;
#pragma unroll
            for (int w = 0; w < 8; ++w) sum += sm.part1[w];
            lim = 4.0f * (sum * inv);
            far = mine && !(norm <= lim);
            const bool again = __syncthreads_or(in && far) != 0; // also: the partial sums may be overwritten
            if (!again || round == 5) break;
            in = mine && !far;
            if (!__syncthreads_or(in)) break; // overflow: void below
        }
        float t = far ? 0.0f : norm;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, o));
        if (lane == 0) sm.part1[warp] = t;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < 8; ++w) rho = fmaxf(rho, sm.part1[w]);
        void_sub = lost || !(rho >= RHO_MIN && rho <= RHO_MAX && lim <= 4.0f * RHO_MAX);
    }
    const uint32_t e = (__float_as_uint(rho) >> 23) & 0xFFu;                     // rho in [2^(e - 127), 2^(e - 126))
    const float scale = void_sub ? 1.0f : __uint_as_float((255u - e) << 23);     // rho * scale in [2, 4)
    constexpr int KROW = 16 * SL::STEPS;
    uint16_t row[KROW];
#pragma unroll
    for (int i = 0; i < KROW; ++i) row[i] = 0;
    const uint16_t one = 0x3C00u;
    if (void_sub) {
        // zeros: the rows' operands are zero as well, every column ties
    } else if (!mine || far) {
        row[SL::CONST] = f32_to_f16_bits(4096.0f + 28.0f); // 2048 * 28 = 57344
    } else {
#pragma unroll
        for (int i = 0; i < SD; ++i) {
            const float c = y[i] * scale;
            const uint16_t h = f32_to_f16_bits(-c);
            const uint16_t l = f32_to_f16_bits(-c - __half2float(__ushort_as_half(h)));
            row[i] = row[2 * SD + i] = h;
            row[SD + i] = l;
        }
        if (!COSINE) {
            const float hn = half_norm * scale * scale;
            row[SL::NORM] = f32_to_f16_bits(hn);
            row[SL::NORM + 1] = f32_to_f16_bits(hn - __half2float(__ushort_as_half(row[SL::NORM])));
        }
        row[SL::CONST] = f32_to_f16_bits(4096.0f);
        row[SL::CONST + 1] = one;
    }
    uint4 *o1 = reinterpret_cast<uint4 *>(scratch + OFF_B1) + ((size_t)s * BN + j) * 4, *o2 = reinterpret_cast<uint4 *>(scratch + OFF_B2) + ((size_t)s * BN + j) * 2;
#pragma unroll
    for (int i = 0; i < KROW / 8; ++i) {
        const uint16_t *w = row + 8 * i;
        (i < 4 ? o1[i] : o2[i - 4]) = make_uint4(w[0] | ((uint32_t)w[1] << 16), w[2] | ((uint32_t)w[3] << 16), w[4] | ((uint32_t)w[5] << 16), w[6] | ((uint32_t)w[7] << 16));
    }
    uint16_t *img = reinterpret_cast<uint16_t *>(scratch + OFF_C16) + ((size_t)s * BN + j) * SD;
#pragma unroll
    for (int i = 0; i < SD; i += 4) {
        uint2 w = make_uint2(0u, 0u);
        if (j < k) {
            w.x = f32_to_f16_bits(v[i]) | ((uint32_t)f32_to_f16_bits(v[i + 1]) << 16);
            w.y = f32_to_f16_bits(v[i + 2]) | ((uint32_t)f32_to_f16_bits(v[i + 3]) << 16);
        }
        *reinterpret_cast<uint2 *>(img + i) = w;
    }
    float *sub = scratch + OFF_SUB + (size_t)s * SUB_FLOATS;
    const uint32_t mask = __ballot_sync(0xffffffffu, far && !void_sub);
    if (lane == 0) sub[SUB_MASK + warp] = __uint_as_float(mask);
    const bool any_far = __syncthreads_or(far && !void_sub) != 0;
    if (j == 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) sub[i] = void_sub || i >= SD ? 0.0f : -mu[i % SD]; // (added to the rows)
        sub[SUB_RHO2] = 1.000001f * rho * rho;
        sub[SUB_SCALE] = scale;
        sub[SUB_SCALE2] = scale * scale;
        sub[SUB_FLAGS] = __uint_as_float((void_sub ? SUB_VOID : 0u) | (any_far ? SUB_FAR : 0u) | (lost && !COSINE ? SUB_NAN0 : 0u));
        sub[SUB_LIM] = 0.99999f * lim;
    }
}

template <int SD> __device__ __forceinline__ void read_centroid(float (&v)[SD], const float *cb, int s, int k, int j)
{
    if (j < k) {
        load_centroid<SD>(v, cb + ((size_t)s * k + j) * SD);
    } else {
#pragma unroll
        for (int i = 0; i < SD; ++i) v[i] = 0.0f;
    }
}

template <int SD, bool COSINE> __global__ void __launch_bounds__(BN) pq_operand_b_kernel(const float *cb, int k, float *scratch)
{
    __shared__ OperandSmem<SD> sm;
    float v[SD];
    after_previous_kernel();
    next_kernel_may_start();
    read_centroid<SD>(v, cb, blockIdx.x, k, threadIdx.x);
    write_operand<SD, COSINE>(v, blockIdx.x, k, scratch, sm);
}

} // namespace

bool pq_tc_applicable(const AssignParams &p, int metric)
{
    return (metric == M_SQ || metric == M_EUCLID || metric == M_COSINE) && pq_tc_shape(p.m, p.sd, p.k) && pq_tc_rows(p.n) &&
           p.ld % 4 == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15u) == 0 && (reinterpret_cast<uintptr_t>(p.centroids) & 15u) == 0 &&
           (reinterpret_cast<uintptr_t>(p.out_f16) & 15u) == 0 && (reinterpret_cast<uintptr_t>(p.out_f32) & 15u) == 0;
}

// The tensor kernel computes 128 columns whatever k is, in three launches; the CUDA-core kernels' one takes a time that grows with k.  Multiples
// of four sub-spaces of 8 values stay here for every k.  Where the others meet, k for the CUDA-core kernels' time over this one's (15,000,
// 60,000 and 300,000 rows):
//   8-wide, Euclidean: m 5 .. 30 at k 24: 0.64 .. 0.92, 0.71 .. 1.05, 0.65 .. 1.01; 32: 0.73 .. 1.14, 0.86 .. 1.21, 0.78 .. 1.18;
//       40: 0.83 .. 1.21, 1.04 .. 1.38, 0.92 .. 1.34 (m 13, 300,000 rows, k 16: 92 us there, 172 here; k 64: 227 and 173)
//   8-wide, cosine: k 16: 0.63 .. 0.98, 0.80 .. 1.31, 0.97 .. 1.63; 24: 0.79 .. 1.23, 1.04 .. 1.70, 1.21 .. 2.04
//   4-wide, m 4 .. 6, Euclidean: k 32: 0.68 .. 0.93, 0.74 .. 0.91, 0.91 .. 1.37; 40: 0.76 .. 0.93, 0.83 .. 0.99, 1.02 .. 1.48 (the last of
//       each is m 4, whose group is full: 1.0 from k 2 on with 300,000 rows); cosine: k 24: 0.77 .. 1.04, 0.82 .. 1.14, 1.33 .. 1.81
//   4-wide, m from 7 on: below 200,000 pairs (m 7 .. 13, 15,000 rows) k 16: 0.79 .. 1.07, 32: 0.89 .. 1.21, cosine k 16: 0.99 .. 1.20;
//       above, every k of the range is faster here (m 16: 1.15 .. 2.4; m 9, 60,000 rows, k 16: 0.95)
// Training passes are faster here for every k (2 .. 64, 30,000 and 300,000 rows: 0.97 .. 2.2).
bool pq_tc_encode_pays(const AssignParams &p, int metric)
{
    if (p.sd == 8) return p.m % 4 == 0 || p.k >= (metric == M_COSINE ? 20 : 36);
    const bool few = p.n * (unsigned long long)p.m < 200000u || p.m == 5 || p.m == 6 || (p.m == 4 && p.n < 150000u);
    return !few || p.k >= (metric == M_COSINE ? 24 : 40);
}

size_t pq_tc_scratch_floats() { return SCRATCH_FLOATS; }
size_t pq_tc_stats_offset_floats() { return OFF_STATS; }
size_t pq_tc_consts_offset_floats() { return OFF_SUB; }
size_t pq_tc_code_bytes(size_t n, size_t m) { return n * m; }

struct PqMaps {
    CUtensorMap x, b1, b2;
};

template <int SD, bool TRAIN, int METRIC, bool WIDE, int DUMP = 0>
static void launch_w(CudaDevice &dev, const PqMaps &mp, const PqTcParams &q, unsigned grid)
{
    auto kernel = pq_tc_kernel<SD, TRAIN, METRIC, WIDE, DUMP>;
    constexpr size_t smem = PQ_TC_SMEM<SD>;
    static std::atomic<unsigned long long> configured{0}; // bit d: the attribute has been set on device d (it is per device and sticky)
    const unsigned long long bit = 1ull << (dev.device() & 63);
    if (!(configured.load(std::memory_order_relaxed) & bit)) {
        VQB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured.fetch_or(bit, std::memory_order_relaxed);
    }
    KernelScope ks(dev, TRAIN ? "assign_train" : "pq_encode");
    launch_following(kernel, grid, NTHREADS, smem, dev.stream(), mp.x, mp.b1, mp.b2, q);
    dev.count_launch();
}

template <int SD, bool TRAIN, int METRIC> static void launch_t(CudaDevice &dev, const PqMaps &mp, const PqTcParams &q, unsigned grid)
{
    if (q.a.k > 128) launch_w<SD, TRAIN, METRIC, true>(dev, mp, q, grid);
    else launch_w<SD, TRAIN, METRIC, false>(dev, mp, q, grid);
}

template <int SD> static void launch_expand(CudaDevice &dev, const AssignParams &p, const uint16_t *c16)
{
    const size_t table = (size_t)p.m * BN * SD * sizeof(uint16_t);
    const bool in_smem = table <= 200u * 1024u;
    auto kernel = in_smem ? pq_expand_kernel<SD, true> : pq_expand_kernel<SD, false>;
    static std::atomic<unsigned long long> configured{0};
    const unsigned long long bit = 1ull << (dev.device() & 63);
    if (!(configured.load(std::memory_order_relaxed) & bit)) {
        VQB_CUDA_CHECK(cudaFuncSetAttribute(pq_expand_kernel<SD, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        configured.fetch_or(bit, std::memory_order_relaxed);
    }
    const unsigned long long pairs = p.n * (unsigned long long)p.m;
    const unsigned per_sm = in_smem ? (unsigned)std::min<size_t>(4, 200u * 1024u / table) : 4u;
    const unsigned grid = (unsigned)std::min<unsigned long long>((pairs + 511) / 512, (unsigned long long)dev.sm_count() * per_sm);
    KernelScope ks(dev, "pq_expand");
    launch_following(kernel, grid, 512, in_smem ? table : 0, dev.stream(), reinterpret_cast<const uint8_t *>(p.codes), pairs, p.m, p.k, c16, p.centroids, p.out_f16, p.out_codes, p.out_f32);
    dev.count_launch();
}

template <int SD> static void launch_sd(CudaDevice &dev, const PqMaps &mp, const PqTcParams &q, unsigned grid, int metric, bool train, const uint16_t *c16)
{
    if (q.dbg_frames) { // T itself, and nothing else
        if (metric == M_COSINE) launch_w<SD, false, M_COSINE, true, 2>(dev, mp, q, grid);
        else launch_w<SD, false, M_SQ, true, 2>(dev, mp, q, grid);
        return;
    }
    if (q.dbg_scores) launch_w<SD, false, M_SQ, true, 1>(dev, mp, q, grid);
    if (train) {
        launch_t<SD, true, M_SQ>(dev, mp, q, grid);
        return;
    }
    if (metric == M_EUCLID) launch_t<SD, false, M_EUCLID>(dev, mp, q, grid);
    else if (metric == M_COSINE) launch_t<SD, false, M_COSINE>(dev, mp, q, grid);
    else launch_t<SD, false, M_SQ>(dev, mp, q, grid);
    if (q.a.out_f16 || q.a.out_codes || q.a.out_f32) launch_expand<SD>(dev, q.a, c16); // else the caller wants the one-byte codes
}

void launch_pq_operand_b(CudaDevice &dev, const float *centroids, int m, int k, int sd, bool cosine, float *scratch)
{
    KernelScope ks(dev, "pq_operand_b");
    auto kernel = sd == 4 ? (cosine ? pq_operand_b_kernel<4, true> : pq_operand_b_kernel<4, false>) : (cosine ? pq_operand_b_kernel<8, true> : pq_operand_b_kernel<8, false>);
    launch_following(kernel, m, BN, 0, dev.stream(), centroids, k, scratch);
    dev.count_launch();
}

PqTcMaps pq_tc_make_maps(const float *scratch)
{
    PqTcMaps maps;
    maps.b1 = make_tensor_map_2d(reinterpret_cast<const uint16_t *>(scratch + OFF_B1), 32, (unsigned long long)MAXM * BN, 32, BN, CU_TENSOR_MAP_SWIZZLE_64B);
    maps.b2 = make_tensor_map_2d(reinterpret_cast<const uint16_t *>(scratch + OFF_B2), 16, (unsigned long long)MAXM * BN, 16, BN, CU_TENSOR_MAP_SWIZZLE_32B);
    return maps;
}

void launch_pq_tc(CudaDevice &dev, const AssignParams &p, int metric, bool train, size_t code_bytes, const PqTcBuffers &b)
{
    if (train && code_bytes != 1) throw Error(100, "pq tensor path: one-byte codes expected for k <= 256");
    if (b.prepare_operand) launch_pq_operand_b(dev, p.centroids, p.m, p.k, p.sd, metric == M_COSINE, b.scratch);
    PqMaps mp;
    mp.b1 = b.maps->b1, mp.b2 = b.maps->b2;
    // the rows as they lie: a box is one tile of a group's columns
    mp.x = make_tensor_map_2d(p.x, (unsigned long long)p.m * p.sd, p.n, 4 * p.sd, BM, p.sd == 8 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, p.ld);
    PqTcParams q = {};
    q.a = p;
    if (!train) q.a.codes = b.codes;
    q.sub = b.scratch + OFF_SUB;
    q.stats = reinterpret_cast<unsigned long long *>(b.scratch + OFF_STATS);
    q.error = b.error_word;
    q.dbg_scores = b.dbg_scores;
    q.dbg_frames = b.dbg_frames;
    // one CTA per SM, shared out among the groups of four sub-spaces by what they hold: the last one may have fewer than four
    const unsigned long long tiles = (p.n + BM - 1) / BM;
    const unsigned ngroups = ((unsigned)p.m + 3) / 4;
    unsigned left = (unsigned)std::max(dev.sm_count(), (int)ngroups), subs = (unsigned)p.m, at = 0;
    for (unsigned g = 0; g < ngroups; ++g) {
        const unsigned here = std::min(4u, (unsigned)p.m - 4 * g);
        const unsigned share = std::max(1u, std::min((left * here + subs / 2) / subs, left - (ngroups - 1 - g)));
        q.first[g] = (uint16_t)at;
        at += (unsigned)std::min<unsigned long long>(tiles, share);
        left -= share;
        subs -= here;
    }
    q.first[ngroups] = (uint16_t)at;
    const uint16_t *c16 = reinterpret_cast<const uint16_t *>(b.scratch + OFF_C16);
    if (p.sd == 4) launch_sd<4>(dev, mp, q, at, metric, train, c16);
    else launch_sd<8>(dev, mp, q, at, metric, train, c16);
}

// ------------------------------------------------------------------------------------------------
// Centroid update of one k-means iteration for the shapes this file serves, in one launch (one CTA per sub-space, thread j =
// cluster j): centroid = sum / count (src/vector.rs:315-316), the operand-B row, binary16 image and constants the next
// assignment pass needs, the iteration's flags for the host, and the sums / counts / flags cleared for the next iteration.
// ------------------------------------------------------------------------------------------------
template <int SD>
__global__ void __launch_bounds__(BN) pq_update_centroids_kernel(float *sums, uint32_t *counts, uint32_t *moved, int counts_f32, const uint32_t *active,
                                                                 int k, float *centroids, float *scratch, StatusPage sp, const PeerView pv)
{
    constexpr int V = SD / 4;
    __shared__ OperandSmem<SD> sm;
    const int s = blockIdx.x, j = threadIdx.x;
    after_previous_kernel();
    next_kernel_may_start();
    const bool act = !active || active[s] != 0;
    const bool direct = pv.world > 1; // the parts of all ranks are added here, in rank order (peer_exchange.cuh)
    peer_arrive_and_wait(pv);
    uint32_t mv_parts[VQB_MAX_PEERS]; // the ranks' "some row moved" words of this sub-space: requested now, used at the end
#pragma unroll
    for (int q = 0; q < VQB_MAX_PEERS; ++q) mv_parts[q] = (direct && j == 0 && q < pv.world) ? peer_ld(pv.words[q] + pv.off_moved + s) : 0u;
    bool empty = false;
    if (act) {
        float v[SD];
#pragma unroll
        for (int i = 0; i < SD; ++i) v[i] = 0.0f;
        if (j < k) {
            const size_t cj = (size_t)s * k + j;
            float4 *cp = reinterpret_cast<float4 *>(centroids + cj * SD);
            float4 *sp4 = reinterpret_cast<float4 *>(sums + cj * SD);
            float4 a[V];
            float cf;
            if (direct) {
                // Every peer load is issued before the first one is used.  A warp stops at the first instruction that needs a
                // pending load, so "load rank q, add, load rank q + 1" pays one NVLink round trip (about 2 us) per rank:
                // 30 us of a 44 us kernel at eight ranks.  The parts are then added in rank order as before.
                float4 part[VQB_MAX_PEERS][V];
                uint32_t pc[VQB_MAX_PEERS];
#pragma unroll
                for (int q = 0; q < VQB_MAX_PEERS; ++q) {
                    pc[q] = 0u;
#pragma unroll
                    for (int i = 0; i < V; ++i) part[q][i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (q < pv.world) {
                        const uint32_t *w = pv.words[q];
#pragma unroll
                        for (int i = 0; i < V; ++i) part[q][i] = peer_ld4(w + cj * SD + 4 * i);
                        pc[q] = peer_ld(w + pv.off_counts + cj);
                    }
                }
                uint32_t cnt = pc[0];
#pragma unroll
                for (int i = 0; i < V; ++i) a[i] = part[0][i];
#pragma unroll
                for (int q = 1; q < VQB_MAX_PEERS; ++q) {
                    if (q < pv.world) {
                        cnt += pc[q];
#pragma unroll
                        for (int i = 0; i < V; ++i) {
                            a[i].x = __fadd_rn(a[i].x, part[q][i].x), a[i].y = __fadd_rn(a[i].y, part[q][i].y);
                            a[i].z = __fadd_rn(a[i].z, part[q][i].z), a[i].w = __fadd_rn(a[i].w, part[q][i].w);
                        }
                    }
                }
                cf = __uint2float_rn(cnt);
                float4 *st4 = reinterpret_cast<float4 *>(pv.stale + cj * SD);
#pragma unroll
                for (int i = 0; i < V; ++i) st4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                pv.stale[pv.off_counts + cj] = 0u;
            } else {
                const uint32_t cw = counts[cj];
                cf = counts_f32 ? __uint_as_float(cw) : __uint2float_rn(cw);
#pragma unroll
                for (int i = 0; i < V; ++i) a[i] = sp4[i];
            }
            if (cf != 0.0f) {
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    a[i] = make_float4(__fdiv_rn(a[i].x, cf), __fdiv_rn(a[i].y, cf), __fdiv_rn(a[i].z, cf), __fdiv_rn(a[i].w, cf));
                    cp[i] = a[i];
                    if (!direct) sp4[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                if (!direct) counts[cj] = 0u;
            } else { // an empty cluster keeps its centroid until the host re-seeds it (src/utils.rs:99-101)
                empty = true;
#pragma unroll
                for (int i = 0; i < V; ++i) a[i] = cp[i];
            }
#pragma unroll
            for (int i = 0; i < V; ++i) v[4 * i] = a[i].x, v[4 * i + 1] = a[i].y, v[4 * i + 2] = a[i].z, v[4 * i + 3] = a[i].w;
        }
        write_operand<SD, false>(v, s, k, scratch, sm);
    }
    // flags of this sub-space for the host: 8 bitmap words (bit = cluster without rows) and the "some row moved" word
    const uint32_t bits = __ballot_sync(0xffffffffu, empty);
    if ((j & 31) == 0 && (uint32_t)(j >> 5) < sp.words_per_subspace) sp.put(sp.idx_bitmap(s, j >> 5), bits);
    if (j == 0) {
        uint32_t mv = 0u;
        if (direct) {
#pragma unroll
            for (int q = 0; q < VQB_MAX_PEERS; ++q) mv |= mv_parts[q];
            pv.stale[pv.off_moved + s] = 0u;
        } else {
            mv = moved[s];
            moved[s] = 0u;
        }
        sp.put(sp.idx_moved(s), act ? mv : 0u);
        if (s == 0) sp.put_error();
    }
}

void launch_pq_update_centroids(CudaDevice &dev, int m, int k, int sd, float *sums, uint32_t *counts, uint32_t *moved, bool counts_f32,
                                const uint32_t *active, float *centroids, float *scratch, const StatusPage &sp, const PeerView &pv)
{
    KernelScope ks(dev, "update_centroids");
    auto kernel = sd == 4 ? pq_update_centroids_kernel<4> : pq_update_centroids_kernel<8>;
    launch_following(kernel, m, BN, 0, dev.stream(), sums, counts, moved, counts_f32 ? 1 : 0, active, k, centroids, scratch, sp, pv);
    dev.count_launch();
}

} // namespace vqb
