// rvq_tc.cu -- the residual encoder (src/rvq.rs:171-215) with all its stages in one kernel, for the shapes of the tensor-core path.
//
// A CTA takes 128 rows through every stage: the residuals and the sums of the chosen centroids stay in registers (a warp has eight rows, a
// lane four dimensions of each), what goes to memory is the input once and the results once.  Per stage
//   1. the residuals' image (two binary16 parts, see dense_tc.cu) goes to shared memory as operand A,
//   2. one thread issues the MMAs against the stage's codebook image, which TMA has brought into shared memory (the next stage's
//      follows as soon as these MMAs are done): D_j = v.c_j - |c_j|^2/2 in tensor memory,
//   3. sixteen warps look at the 128 x 256 scores: largest one per row, then a mask of the centroids within the error bound,
//   4. rows with one candidate have their code; the others' candidates are evaluated with the reference's serial f32 chain: up to
//      eight by the row's own warp (whole centroids loaded, one lane per candidate adding up), more by all warps together against all
//      centroids, a row with a value that is not finite not at all (no distance is below +inf: centroid 0),
//   5. residual, running sum, norm against epsilon.
// The multi-launch path that this replaces wrote residual, image and norms of every row in every stage (1 KB a row).
//
// Scales.  Codebooks have a frame from their own centroids (mu: their mean, beta: a power of two that brings the largest norm to
// [32, 64)); a row's residual is taken relative to the same mu and scaled by its own power of two alpha, so that its parts are as exact as
// binary16 has them whatever the codebook looks like.  The half norms enter by a last K = 8 step with the factor rho = alpha / beta as
// the row's operand: D is in units of alpha beta.  Bound as in dense_tc.cu, in these units:
//   E = 7e-6 |v| |c| + 4e-7 (|v| + |c|) + 6e-7 rho |c|^2     (|v| = alpha |x - mu|, |c| = beta max |c_j - mu|)
//   limit = S_min + 2 E + 1.05 (dim + 6) 2^-24 (|v|^2 / rho + 2 S_min + 2 E)
// alpha is kept within 2^-60 .. 2^20 of beta: |v|^2 / rho and rho |c|^2 stay far inside f32.
//
// Measured (us a call, before -> now; 128 values, 256 centroids, 8 stages): 4,999 rows 193 -> 66, 12,000 rows 466 -> 83, 40,000 rows 912 -> 200,
// 1,000,000 rows 16,200 -> 3,340 (in these codebooks dozens of centroids are equal; 2 stages, few equal ones: 48 -> 29, 102 -> 35, 125 -> 66, 1121
// -> 973); 1,000,000 x 64: 2505 -> 2221, x 32: 1589 -> 1507; 1,000,000 x 61, 4 stages: 1422 -> 1280.  What bounds it is the chain of a stage
// in a CTA, 9,800 cycles with 64 rows and 13,000 with 128: image 1,600 / 2,000, MMAs 3,750 (3,200 of them the tensor core's), scores 1,450 / 2,100,
// codes 650 (3,100 for a warp with a row that is not decided, for which the others wait), the centroids' way from L2 2,000, norms 450.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "assign_generic.cuh"
#include "cuda_device.hpp"
#include "dense_image.cuh"
#include "dense_tc.hpp"
#include "kernels_common.cuh"
#include "tma_host.hpp"
#include "umma.cuh"

namespace vqb {

namespace {

constexpr int BM = 128, CHUNK = 64;      // rows of an operand tile; binary16 values of a 128-byte operand row
constexpr int NT = 512, NWARP = NT / 32; // (128 registers a thread)

// per-stage constants (floats): mu[128], then
constexpr int F_BETA = 128, F_CMAX = 129, F_EXP = 130, F_FLOATS = 132;

struct alignas(8) RvqBarriers {
    unsigned long long bfull, tfull;
    uint32_t tmem_base;
    int abort_flag;
};

struct RvqStagesParams {
    const float *x, *books; // [n][dim], [stages][k][dim]
    unsigned long long n;
    int dim, k, stages, euclid, vec; // vec: rows and centroids are whole 16-byte pieces
    float epsilon;
    float *frames;   // [stages][F_FLOATS]
    uint16_t *image; // [stages][bn][2 * DIMP]
    float *extra;    // [stages][bn][8] operand B of the half norms, as the tile lies in shared memory
    int one;         // a cooperative launch, which lays the codebooks out itself
    int book_vec;    // centroids are whole 16-byte pieces
    uint16_t *out_f16;
    uint32_t *out_codes;
    int *error;
};

template <int BN> struct Shared { // behind the operand tiles
    float part[4][BM];           // largest score of a row in a quarter of the columns
    float vn2[BM], alpha[BM];    // |v|^2 (upper bound), scale of a row
    uint32_t mask[BM][BN / 32];  // candidates
    uint8_t nan0[BM];
    uint8_t open[BM];             // rows with many candidates, in any order
    uint32_t n_open;
    unsigned long long least[BM]; // of each of them: bits of the smallest distance so far (never negative: ordered like the numbers), its centroid
    RvqBarriers bars;
};

template <int BN> constexpr uint32_t BOOK_CHUNK = BN * 128; // bytes of a chunk of a codebook image
template <int KS, int BN> constexpr size_t stages_smem()
{
    constexpr size_t kchunks = (2 * KS + 3) / 4;
    return 1024 + kchunks * (BOOK_CHUNK<BN> + BM * 128) + (BN + BM) * 32 + sizeof(Shared<BN>);
}

__device__ __forceinline__ void umma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate, bool tf32)
{
    if (tf32)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

// Sums over the L lanes of a row group of N values at once (N <= 8, N <= L): of its lanes, L / N for each value, group i gets the sum of a[i]
template <int N, int L> __device__ __forceinline__ float sum_rows(const float (&a)[N], int lane)
{
    if constexpr (N == 1) {
        float d = a[0];
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
        return d;
    } else {
        const bool up = (lane & (L / 2)) != 0;
        float b[N / 2];
#pragma unroll
        for (int i = 0; i < N / 2; ++i) b[i] = (up ? a[i + N / 2] : a[i]) + __shfl_xor_sync(0xffffffffu, up ? a[i] : a[i + N / 2], L / 2);
        return sum_rows<N / 2, L / 2>(b, lane);
    }
}

// the reference's serial sum, four terms on
__device__ __forceinline__ void square_differences(float &d, const float4 &x, const float4 &c)
{
    const float e0 = __fsub_rn(x.x, c.x), e1 = __fsub_rn(x.y, c.y), e2 = __fsub_rn(x.z, c.z), e3 = __fsub_rn(x.w, c.w);
    d = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(d, __fmul_rn(e0, e0)), __fmul_rn(e1, e1)), __fmul_rn(e2, e2)), __fmul_rn(e3, e3));
}

// exponent that brings a norm, given its square, to [32, 64)
__device__ __forceinline__ int scale_exponent(float square) { return 5 - (((int)((__float_as_uint(square) >> 23) & 0xFFu) - 127) >> 1); }
__device__ __forceinline__ float power_of_two(int e) { return __uint_as_float((uint32_t)(127 + e) << 23); }

__device__ __forceinline__ void load4(float (&v)[4], const float *p, int lane, int dim, bool vec, bool in)
{
    if (vec) {
        const float4 t = in && 4 * lane < dim ? __ldg(reinterpret_cast<const float4 *>(p) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = in && 4 * lane + e < dim ? __ldg(p + 4 * lane + e) : 0.0f;
    }
}

// two values in two binary16 parts each
__device__ __forceinline__ void split_pair(float v0, float v1, uint32_t &h, uint32_t &l)
{
    const __half2 hh = __floats2half2_rn(v0, v1), ll = __floats2half2_rn(v0 - __low2float(hh), v1 - __high2float(hh));
    h = *reinterpret_cast<const uint32_t *>(&hh), l = *reinterpret_cast<const uint32_t *>(&ll);
}

template <int W> struct BookShared {
    alignas(16) float sum[W][128];
    alignas(16) float mu[128];
    alignas(16) uint32_t hash[256];
    uint32_t first[256], count, big, hmax;
};

// Frame, image and half norms of a stage's codebook, by a whole CTA.  A centroid that equals one before it in every value never wins
// (equal distances, strict '<' in ascending order), so its column is like one beyond k: training on few rows leaves dozens of equal
// centroids, zeros mostly, and every row that chose one of them would be left to the exact evaluation with all of them.
// All of it is in registers from one trip to memory on (a warp has every THREADS / 32nd centroid, a lane four dimensions of each).
template <int THREADS>
__device__ __forceinline__ void make_book(BookShared<THREADS / 32> &s, const float *books, int st, int k, int dim, int dimp, int bn, bool vec, float *frames, uint16_t *image, float *extra)
{
    constexpr int W = THREADS / 32, C = 256 / W; // centroids of a warp
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float *book = books + (size_t)st * k * dim;
    if (tid == 0) s.count = s.big = s.hmax = 0u;
    if (tid < 256) s.first[tid] = tid;
    float v[C][4], sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < C; ++i) load4(v[i], book + (size_t)(warp + W * i) * dim, lane, dim, vec, warp + W * i < k);
    __syncthreads();
    uint32_t count = 0;
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int j = warp + W * i;
        const float big = fmaxf(fmaxf(fabsf(v[i][0]), fabsf(v[i][1])), fmaxf(fabsf(v[i][2]), fabsf(v[i][3])));
        const bool nan = !(v[i][0] + v[i][1] + v[i][2] + v[i][3] == v[i][0] + v[i][1] + v[i][2] + v[i][3]);
        if (j < k && __all_sync(0xffffffffu, big < 1e37f && !nan)) { // what is not finite has no say
            ++count;
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[e] += v[i][e];
        }
        uint32_t hash = 0;
#pragma unroll
        for (int e = 0; e < 4; ++e) hash = (hash ^ __float_as_uint(v[i][e] + 0.0f)) * 0x9E3779B1u; // (-0 + 0 = +0)
        hash = __reduce_add_sync(0xffffffffu, hash * (2u * lane + 1u));
        if (lane == 0) s.hash[j] = hash;
    }
    *reinterpret_cast<float4 *>(&s.sum[warp][4 * lane]) = make_float4(sum[0], sum[1], sum[2], sum[3]);
    if (lane == 0) atomicAdd(&s.count, count);
    __syncthreads();
    float *fr = frames + (size_t)st * F_FLOATS;
    if (tid < 128) {
        float t = 0.0f;
#pragma unroll
        for (int w = 0; w < W; ++w) t += s.sum[w][tid];
        const float mu = t / fmaxf((float)s.count, 1.0f);
        s.mu[tid] = fabsf(mu) < VQB_DENSE_INF ? mu : 0.0f;
        fr[tid] = s.mu[tid];
    }
    {
        const int j = tid & 255, from = (tid >> 8) * (256 / (THREADS / 256)); // THREADS / 256 threads look for the first centroid with the same hash
        const uint32_t mine = s.hash[j];
        int first = 256;
#pragma unroll 4
        for (int i = 256 / (THREADS / 256) - 4; i >= 0; i -= 4) {
            const uint4 h = *reinterpret_cast<const uint4 *>(&s.hash[from + i]);
            first = h.w == mine ? from + i + 3 : first, first = h.z == mine ? from + i + 2 : first;
            first = h.y == mine ? from + i + 1 : first, first = h.x == mine ? from + i : first;
        }
        if (j < k && first < j) atomicMin(&s.first[j], (uint32_t)first);
    }
    __syncthreads();
    const float4 mu = *reinterpret_cast<const float4 *>(&s.mu[4 * lane]);
    uint32_t gone = 0; // bit i: no centroid, or one that cannot win
    float a[C];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int j = warp + W * i;
        bool same = j >= k;
        if (!same && s.first[j] < (uint32_t)j) { // equal indeed?
            float w[4];
            load4(w, book + (size_t)s.first[j] * dim, lane, dim, vec, true);
            same = __all_sync(0xffffffffu, v[i][0] == w[0] && v[i][1] == w[1] && v[i][2] == w[2] && v[i][3] == w[3]);
        }
        gone |= (same ? 1u : 0u) << i;
        v[i][0] -= mu.x, v[i][1] -= mu.y, v[i][2] -= mu.z, v[i][3] -= mu.w;
        a[i] = fmaf(v[i][0], v[i][0], fmaf(v[i][1], v[i][1], fmaf(v[i][2], v[i][2], v[i][3] * v[i][3])));
    }
    constexpr int LPC = 32 / C;
    const float sq = sum_rows<C, 32>(a, lane); // of centroid lane / LPC
    const bool here = !(gone >> (lane / LPC) & 1u);
    if (lane % LPC == 0 && here && sq < VQB_DENSE_INF) atomicMax(&s.big, __float_as_uint(sq));
    __syncthreads();
    const int eb = s.big ? min(max(scale_exponent(__uint_as_float(s.big)), -60), 60) : 0;
    const float beta = power_of_two(eb);
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int j = warp + W * i;
        uint32_t h[2], l[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) split_pair(gone >> i & 1u ? 0.0f : v[i][2 * e] * beta, gone >> i & 1u ? 0.0f : v[i][2 * e + 1] * beta, h[e], l[e]);
        if (j < bn && 4 * lane < dimp) {
            uint16_t *o = image + ((size_t)st * bn + j) * 2 * dimp + 4 * lane;
            *reinterpret_cast<uint2 *>(o) = make_uint2(h[0], h[1]);
            *reinterpret_cast<uint2 *>(o + dimp) = make_uint2(l[0], l[1]);
        }
    }
    const int j = warp + W * (lane / LPC);
    if (lane % LPC == 0 && j < bn) {
        const float hn = 0.5f * beta * beta * sq;
        if (here) atomicMax(&s.hmax, __float_as_uint(fmaxf(hn, 0.0f))); // (NaN counts as 0)
        const bool pad = !here || !(hn < VQB_DENSE_INF);
        const float hh = pad ? 1e30f : tf32_round(hn), hl = pad ? 0.0f : tf32_round(hn - hh);
        float *xp = extra + ((size_t)st * bn + j) * 8;
        const int sw = ((j >> 2) & 1) * 4; // 32B swizzle: the two 16-byte halves of a row swap when bit 2 of the row is set
        *reinterpret_cast<float4 *>(xp + sw) = make_float4(-hh, -hl, 0.0f, 0.0f);
        *reinterpret_cast<float4 *>(xp + (4 - sw)) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    __syncthreads();
    if (tid == 0) {
        fr[F_BETA] = beta;
        fr[F_CMAX] = sqrtf(2.0f * __uint_as_float(s.hmax)) * 1.00002f;
        fr[F_EXP] = __int_as_float(eb);
    }
}

// KS: K = 16 steps of one part of an image; BN: columns, 128 or 256; ROWS: rows of a warp, 8, or 4 where the rows are so few that half a tile
// of them per SM leaves SMs over.  L lanes share a row (four dimensions each), so that a warp has 32 / L rows in an instruction.
template <int KS, int BN, int ROWS>
__global__ void __launch_bounds__(NT, 1) rvq_stages_kernel(const __grid_constant__ CUtensorMap map_b, const __grid_constant__ RvqStagesParams P)
{
    constexpr int kchunks = (2 * KS + 3) / 4, DIMP = 16 * KS, COLS = BN / 4, WORDS = BN / 32, TILE = NWARP * ROWS;
    constexpr int L = KS <= 2 ? 8 : KS <= 4 ? 16 : 32, RL = 32 / L, NI = ROWS / RL; // rows side by side, registers for rows
    constexpr int LPR = 32 / ROWS, LWORDS = WORDS > LPR ? WORDS / LPR : 1; // lanes that have a row's state, mask words that each looks at
    constexpr uint32_t IDESC_F16 = (1u << 4) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
    constexpr uint32_t IDESC_TF32 = IDESC_F16 | (2u << 7) | (2u << 10);
    extern __shared__ unsigned char smem_raw[];
    unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *b_smem = base;                                                  // the stage's codebook: kchunks x BN rows of 128 bytes
    unsigned char *a_smem = b_smem + (size_t)kchunks * BOOK_CHUNK<BN>;     // the rows' images: kchunks x 128 rows of 128 bytes
    unsigned char *bx_smem = a_smem + (size_t)kchunks * BM * 128;                  // half norms: BN rows of 32 bytes
    unsigned char *ax_smem = bx_smem + BN * 32;                                    // rho, rho: 128 rows of 32 bytes
    Shared<BN> &sh = *reinterpret_cast<Shared<BN> *>(ax_smem + BM * 32);
    volatile int *abort_flag = &sh.bars.abort_flag;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int dim = P.dim, k = P.k;
    const bool vec = P.vec != 0;

    if (tid == 0) {
        mbar_init(&sh.bars.bfull, 1);
        mbar_init(&sh.bars.tfull, 1);
        sh.bars.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sh.bars.tmem_base)), "r"((uint32_t)BN) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sh.bars.tmem_base;
    after_previous_kernel();
    next_kernel_may_start();

    if constexpr (TILE < BM) { // the operand rows that no row uses
        for (int i = tid; i < kchunks * (BM - TILE) * 8; i += NT) reinterpret_cast<uint4 *>(a_smem + (i / ((BM - TILE) * 8)) * (BM * 128) + TILE * 128)[i % ((BM - TILE) * 8)] = make_uint4(0u, 0u, 0u, 0u);
        for (int i = tid; i < (BM - TILE) * 2; i += NT) reinterpret_cast<uint4 *>(ax_smem + TILE * 32)[i] = make_uint4(0u, 0u, 0u, 0u);
    }
    bool ok = true;
    if (P.one) { // the codebooks' images by the first CTAs, then all wait for them at the launch's own barrier
        BookShared<NWARP> &scratch = *reinterpret_cast<BookShared<NWARP> *>(b_smem);
        for (int st = blockIdx.x; st < P.stages; st += gridDim.x) {
            make_book<NT>(scratch, P.books, st, k, dim, DIMP, BN, P.book_vec != 0, P.frames, P.image, P.extra);
            asm volatile("fence.proxy.async;" ::: "memory"); // TMA reads them
            __syncthreads();
        }
        cooperative_groups::this_grid().sync();
        asm volatile("fence.proxy.async;" ::: "memory");
    }
    auto load_book = [&](int st) { // by one thread
        mbar_expect_tx(&sh.bars.bfull, kchunks * BOOK_CHUNK<BN> + BN * 32);
        for (int kc = 0; kc < kchunks; ++kc) tma_load_2d(b_smem + (size_t)kc * BOOK_CHUNK<BN>, &map_b, kc * CHUNK, st * BN, &sh.bars.bfull);
        bulk_load_1d(bx_smem, P.extra + (size_t)st * BN * 8, BN * 32, &sh.bars.bfull);
    };
    const unsigned long long n_tiles = (P.n + TILE - 1) / TILE;
    uint32_t it = 0, loads = 0; // stages so far (parity: that of both barriers); codebooks asked for
    if (tid == 0 && blockIdx.x < n_tiles) load_book(0), ++loads;

    const int first = warp * ROWS, piece = lane % L, side = lane / L; // the warp's first row; this lane's dimensions 4 piece .. 4 piece + 3 of rows i RL + side
    const int sub = lane % LPR, own_row = piece / LPR * RL + side;     // the row whose state this lane (one of LPR) has
    unsigned char *const own = a_smem + first * 128; // this warp's rows of an operand chunk: scratch while no image is in them
    auto row_of = [&](int l) { return l % L / LPR * RL + l / L; };
    float v[NI][4], q[NI][4];
    auto pick_row = [&](float (&t)[4], int r) { // to all lanes (r is the same for the warp; registers cannot be indexed)
#pragma unroll
        for (int e = 0; e < 4; ++e) t[e] = v[0][e];
#pragma unroll
        for (int i = 1; i < NI; ++i)
            if (r / RL == i) t[0] = v[i][0], t[1] = v[i][1], t[2] = v[i][2], t[3] = v[i][3];
        if (RL > 1) {
#pragma unroll
            for (int e = 0; e < 4; ++e) t[e] = __shfl_sync(0xffffffffu, t[e], r % RL * L + piece);
        }
    };
    constexpr int PER = ROWS * 128 / (4 * DIMP); // scratch rows in them
    // Rows with more candidates than FEW_CANDIDATES (a batch of four takes a warp 2,900 cycles): PASS of them at a time against all centroids, PL
    // pieces of 16 bytes at a time; a warp has PASS_ROWS of them and 64 centroids, two a lane.  us a call, 8 stages of 256, 128 wide, every row
    // by its own warp / now / with direct.cu and resolve.cu: 1,500 rows far from all centroids 3,428 / 455 / 563, families of 32 centroids a
    // rounding apart 450 / 358 / 204, values that are not finite 4,394 / 107 / 569, in 1 % of the rows 768 / 72 / 283; 40,000 rows 17,652 / 3,043 / 19,329,
    // 2,190 / 2,080 / 4,420, 23,828 / 428 / 19,675, 2,291 / 215 / 3,816.  4 stages of 64 wide, 1,500 rows far 1,013 / 151 / 135.  Rows that are
    // decided: 4,999 x 128 67.1 / 68.6, 40,000 210 / 207 (this code in line with the rest instead of behind __builtin_expect 215).
    constexpr int FEW_CANDIDATES = 8, PASS_ROWS = ROWS == 8 ? 4 : 8, PASS = PASS_ROWS * NWARP * 2 / WORDS, PL = KS == 8 ? 8 : kchunks > 1 ? 4 : 2, PC = (PL * BN + NT - 1) / NT;
    static_assert((4 * KS) % PL == 0 && PASS * 4 * DIMP + PL * BN * 16 <= kchunks * BM * 128, "rows and centroids of a pass lie in operand A");
    constexpr int BATCH = PER * kchunks < 4 ? PER * kchunks : 4; // candidates at a time (eight: 116 bytes of registers spilled, 5 % slower)
    auto scratch = [&](int b, int p) { // 16-byte piece p of scratch row b
        return reinterpret_cast<float4 *>(own + (size_t)(b / PER) * (BM * 128) + (b % PER) * (4 * DIMP)) + (p ^ (b & 3));
    };

    auto serial_sum = [&](int b) { // of scratch row b, in ascending order; the next pieces are on their way while one group is added up
        float d = 0.0f;
        float4 e[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) e[i] = *scratch(b, i);
#pragma unroll 1
        for (int p = 4; p <= DIMP / 4; p += 4) {
            float4 f[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) f[i] = *scratch(b, p < DIMP / 4 ? p + i : i);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                d = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(d, e[i].x), e[i].y), e[i].z), e[i].w);
                e[i] = f[i];
            }
        }
        return d;
    };

    for (unsigned long long tile = blockIdx.x; ok && tile < n_tiles; tile += gridDim.x) {
        const unsigned long long row0 = tile * TILE + first;
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const unsigned long long row = row0 + i * RL + side;
            load4(v[i], P.x + row * dim, piece, dim, vec, row < P.n);
            q[i][0] = q[i][1] = q[i][2] = q[i][3] = 0.0f;
        }
        const unsigned long long my_row = row0 + own_row;
        bool live = my_row < P.n;                             // takes part in the stages still
        for (int st = 0; st < P.stages; ++st, ++it) {
            // ---- 1. operand A
            {
                const float *fr = P.frames + (size_t)st * F_FLOATS;
                const float4 m4 = reinterpret_cast<const float4 *>(fr)[piece];
                const float mu[4] = {m4.x, m4.y, m4.z, m4.w};
                const int eb = __float_as_int(fr[F_EXP]);
                float a[NI];
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    a[i] = 0.0f;
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float t = v[i][e] - mu[e];
                        a[i] = fmaf(t, t, a[i]);
                    }
                }
                const float sq = sum_rows<NI, L>(a, lane);
                const int ea = min(max(scale_exponent(sq), eb - 60), eb + 20);
                const float mine = power_of_two(ea), rho = power_of_two(ea - eb);
                if (sub == 0) {
                    const int r = first + own_row;
                    sh.vn2[r] = sq * mine * mine * 1.00001f;
                    sh.alpha[r] = mine;
                    unsigned char *ap = ax_smem + (r >> 3) * 256 + (r & 7) * 32;
                    const int sw = ((r >> 2) & 1) * 16; // 32B swizzle
                    *reinterpret_cast<float4 *>(ap + sw) = make_float4(rho, rho, 0.0f, 0.0f);
                    *reinterpret_cast<float4 *>(ap + (16 - sw)) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
                __syncwarp(); // (the scratch is read)
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    const float alpha = __shfl_sync(0xffffffffu, mine, side * L + i * LPR);
                    uint32_t h[2], l[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) split_pair((v[i][2 * e] - mu[2 * e]) * alpha, (v[i][2 * e + 1] - mu[2 * e + 1]) * alpha, h[e], l[e]);
                    if (4 * piece < DIMP) { // 128B swizzle: 16-byte pieces exchanged by the row's number
                        const int r = i * RL + side, x = (first + r) & 7, hp = 4 * piece, lp = DIMP + 4 * piece;
                        *reinterpret_cast<uint2 *>(own + (hp >> 6) * (BM * 128) + r * 128 + ((((hp & 63) >> 3) ^ x) << 4) + (hp & 4) * 2) = make_uint2(h[0], h[1]);
                        *reinterpret_cast<uint2 *>(own + (lp >> 6) * (BM * 128) + r * 128 + ((((lp & 63) >> 3) ^ x) << 4) + (lp & 4) * 2) = make_uint2(l[0], l[1]);
                    }
                }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic writes -> visible to the MMA's reads
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncthreads();
            if (tid == 0) sh.n_open = 0u;
            // ---- 2. scores
            if (tid == 0 && mbar_wait(&sh.bars.bfull, it & 1u, abort_flag, P.error, 41)) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t ad = smem_desc_sw128(smem_u32(a_smem)), bd = smem_desc_sw128(smem_u32(b_smem));
                auto at = [](int step, uint32_t chunk_bytes) { return (uint64_t)((step >> 2) * (int)(chunk_bytes >> 4) + 2 * (step & 3)); };
#pragma unroll
                for (int j = 0; j < KS; ++j) { // h.ch and h.cl
                    umma(tmem, ad + at(j, BM * 128), bd + at(j, BOOK_CHUNK<BN>), IDESC_F16, j ? 1u : 0u, false);
                    umma(tmem, ad + at(j, BM * 128), bd + at(KS + j, BOOK_CHUNK<BN>), IDESC_F16, 1u, false);
                }
#pragma unroll
                for (int j = 0; j < KS; ++j) // l.ch
                    umma(tmem, ad + at(KS + j, BM * 128), bd + at(j, BOOK_CHUNK<BN>), IDESC_F16, 1u, false);
                umma(tmem, smem_desc_sw32(smem_u32(ax_smem)), smem_desc_sw32(smem_u32(bx_smem)), IDESC_TF32, 1u, true);
                umma_commit(&sh.bars.tfull);
            }
            __syncwarp();
            const bool there = mbar_wait(&sh.bars.tfull, it & 1u, abort_flag, P.error, 42);
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (tid == 0 && there && (st + 1 < P.stages || tile + gridDim.x < n_tiles)) load_book(st + 1 < P.stages ? st + 1 : 0), ++loads;
            // ---- 3. the largest score of each row, then the centroids within the bound
            const int er = 32 * (warp & 3) + lane, quarter = warp >> 2; // this thread's row and columns
            const uint32_t taddr = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + quarter * COLS;
            const bool mine_q = TILE == BM || (warp & 3) < TILE / 32; // (the other quadrants of the accumulator hold no rows)
            uint32_t t[32];
            if (mine_q) {
                float top = __uint_as_float(0xFF800000u);
#pragma unroll
                for (int c = 0; c < COLS; c += 32) {
                    tmem_ld32_issue(taddr + c, t);
                    tmem_wait();
                    if (c == 0 && quarter == 0) sh.nan0[er] = !(__uint_as_float(t[0]) == __uint_as_float(t[0]));
                    float m0 = __uint_as_float(t[0]), m1 = __uint_as_float(t[1]);
#pragma unroll
                    for (int i = 2; i < 30; i += 4) {
                        m0 = max3f(m0, __uint_as_float(t[i]), __uint_as_float(t[i + 1]));
                        m1 = max3f(m1, __uint_as_float(t[i + 2]), __uint_as_float(t[i + 3]));
                    }
                    m0 = max3f(m0, __uint_as_float(t[30]), __uint_as_float(t[31]));
                    top = c ? max3f(top, m0, m1) : fmaxf(m0, m1);
                }
                sh.part[quarter][er] = top;
            }
            __syncthreads();
            if (*abort_flag) { // (set before the barrier by whoever gave up: everybody leaves here)
                ok = false;
                break;
            }
            int found = 0; // candidates in this thread's columns
            if (mine_q) {
                const float best = -fmaxf(fmaxf(sh.part[0][er], sh.part[1][er]), fmaxf(sh.part[2][er], sh.part[3][er])); // smallest score
                const float *fr = P.frames + (size_t)st * F_FLOATS;
                const float cmax = fr[F_CMAX], beta = fr[F_BETA], alpha = sh.alpha[er], xn2 = sh.vn2[er];
                const float inv_a = power_of_two(127 - (int)(__float_as_uint(alpha) >> 23)), inv_b = power_of_two(127 - (int)(__float_as_uint(beta) >> 23));
                const float rho = alpha * inv_b, xn = sqrtf(xn2);
                const float e2 = 2.0f * (7e-6f * xn * cmax + 4e-7f * (xn + cmax)) + 1.2e-6f * rho * cmax * cmax;
                const float d_a = fmaxf(xn2 * (beta * inv_a) + 2.0f * best + e2, 0.0f);
                const float limit = best + e2 + 1.05f * (float)(dim + 6) * 5.9604645e-8f * d_a + 2.4e-7f * (fabsf(best) + e2) + 1e-36f * alpha * beta;
                // not to be ranked (NaN / infinity somewhere, a centroid 0 that nothing compares with, distances that could overflow): everything
                const bool scan_all = sh.nan0[er] || !(best == best) || !(limit == limit) || !(fabsf(limit) < VQB_DENSE_INF) ||
                                      !(xn2 * inv_a * inv_a + cmax * inv_b * (cmax * inv_b) < 1e37f);
                const float lim_d = -limit;
#pragma unroll
                for (int c = 0; c < COLS; c += 32) {
                    tmem_ld32_issue(taddr + c, t);
                    tmem_wait();
                    uint32_t m = 0;
#pragma unroll
                    for (int i = 0; i < 32; ++i) m = __funnelshift_l(__float_as_uint(__uint_as_float(t[i]) - lim_d), m, 1);
                    const int lo = quarter * COLS + c;
                    const uint32_t in_range = k >= lo + 32 ? 0xFFFFFFFFu : k > lo ? (1u << (k - lo)) - 1u : 0u;
                    const uint32_t word = (scan_all ? 0xFFFFFFFFu : ~__brev(m)) & in_range;
                    sh.mask[er][lo >> 5] = word;
                    found += __popc(word);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            const bool maybe_many = __syncthreads_or(found > FEW_CANDIDATES / 4); // (more than that in all four quarters: one has more than a fourth)
            // ---- 4. codes: a row's lanes look at its mask
            const float *book = P.books + (size_t)st * k * dim;
            int code = -1;
            {
                int cnt = 0;
#pragma unroll
                for (int w = sub * LWORDS; w < (sub + 1) * LWORDS; ++w) {
                    const uint32_t word = w < WORDS ? sh.mask[first + own_row][w] : 0u;
                    cnt += __popc(word);
                    if (word) code = w * 32 + 31 - __clz(word);
                }
#pragma unroll
                for (int o = LPR / 2; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o), code = max(code, __shfl_xor_sync(0xffffffffu, code, o));
                bool many = false, any_many = false;
                if (__builtin_expect(maybe_many, 0)) {
                    many = live && cnt > FEW_CANDIDATES;
                    any_many = __syncthreads_or(many);
                    // a value that is not finite leaves no distance below +inf: centroid 0
#pragma unroll
                    for (int i = 0; i < NI; ++i) {
                        const bool off = !(fabsf(v[i][0]) < VQB_DENSE_INF && fabsf(v[i][1]) < VQB_DENSE_INF && fabsf(v[i][2]) < VQB_DENSE_INF && fabsf(v[i][3]) < VQB_DENSE_INF);
                        const uint32_t lanes = __ballot_sync(0xffffffffu, off) >> (side * L) & (0xFFFFFFFFu >> (32 - L));
                        if (lanes && piece / LPR == i && many) code = 0, cnt = 1, many = false;
                    }
                }
                uint32_t open = __ballot_sync(0xffffffffu, live && cnt != 1 && !many && sub == 0);
                while (open) {
                    const int r = row_of(__ffs(open) - 1);
                    open &= open - 1;
                    uint32_t word = lane < WORDS ? sh.mask[first + r][lane] : 0u; // what is left of the row's candidates
                    float xr[4];
                    pick_row(xr, r);
                    uint32_t least = 0xFFFFFFFFu; // bits of the smallest distance (never negative: ordered like the numbers)
                    int chosen = 0;               // stays where nothing is below +inf
                    bool stuck = false;
                    for (uint32_t left = __ballot_sync(0xffffffffu, word != 0u); left;) {
                        float c[BATCH][4];
                        int mine = -1, n = 0; // lane b: the b-th candidate of this batch
#pragma unroll
                        for (int b = 0; b < BATCH; ++b) {
                            if (!left) break;
                            const int w = __ffs(left) - 1, j = 32 * w + __shfl_sync(0xffffffffu, __ffs(word) - 1, w);
                            if (lane == w) word &= word - 1;
                            if (lane == b) mine = j;
                            left = __ballot_sync(0xffffffffu, word != 0u);
                            load4(c[b], book + (size_t)j * dim, piece, dim, vec, true);
                            n = b + 1;
                        }
#pragma unroll
                        for (int b = 0; b < BATCH; ++b) {
                            if (b >= n) break;
                            float4 e;
                            e.x = __fsub_rn(xr[0], c[b][0]), e.y = __fsub_rn(xr[1], c[b][1]), e.z = __fsub_rn(xr[2], c[b][2]), e.w = __fsub_rn(xr[3], c[b][3]);
                            e.x = __fmul_rn(e.x, e.x), e.y = __fmul_rn(e.y, e.y), e.z = __fmul_rn(e.z, e.z), e.w = __fmul_rn(e.w, e.w);
                            if (lane < DIMP / 4) *scratch(b, lane) = e; // (beyond dim: zeros, which change no sum of squares)
                        }
                        __syncwarp();
                        float d = serial_sum(lane < n ? lane : 0);
                        if (P.euclid) d = __fsqrt_rn(d);
                        stuck = stuck || __any_sync(0xffffffffu, mine == 0 && !(d == d)); // the reference's scan starts at centroid 0: a NaN there stays
                        const uint32_t u = mine >= 0 && d < VQB_DENSE_INF ? __float_as_uint(d) : 0xFFFFFFFFu, low = __reduce_min_sync(0xffffffffu, u);
                        const int jm = (int)__reduce_min_sync(0xffffffffu, u == low ? (uint32_t)mine : 0xFFFFFFFFu);
                        if (low < least) least = low, chosen = jm; // candidates ascend: an equal distance later on loses
                        __syncwarp();
                    }
                    if (own_row == r) code = stuck ? 0 : chosen;
                }
                if (__builtin_expect(any_many, 0)) { // all warps look at these rows together (the scratch in operand A is free: dense passes below)
                    int place = 0;
                    if (many && sub == 0) {
                        place = (int)atomicAdd(&sh.n_open, 1u);
                        sh.open[place] = (uint8_t)(first + own_row);
                        sh.least[place] = 0xFFFFFFFF00000000ull; // centroid 0 where nothing is below +inf
                    }
                    place = __shfl_sync(0xffffffffu, many ? place : 1 << 20, lane - sub);
                    __syncthreads();
                    const int n_open = (int)sh.n_open;
                    float4 *const rows = reinterpret_cast<float4 *>(a_smem), *const planes = rows + PASS * (DIMP / 4); // [PASS][DIMP / 4], [PL][BN]
                    const int lo = 64 * (warp % (WORDS / 2)), at = PASS_ROWS * (warp / (WORDS / 2)); // this warp's candidates, two a lane, and rows of a pass
                    for (int pass = 0; pass < n_open; pass += PASS) {
#pragma unroll
                        for (int i = 0; i < NI; ++i) {
                            const int pos = __shfl_sync(0xffffffffu, place, side * L + i * LPR) - pass;
                            if (pos >= 0 && pos < PASS && 4 * piece < DIMP) rows[pos * (DIMP / 4) + piece] = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
                        }
                        const int here = min(PASS_ROWS, n_open - pass - at); // (below 1: none)
                        float d[2][PASS_ROWS];
#pragma unroll
                        for (int g = 0; g < PASS_ROWS; ++g) d[0][g] = d[1][g] = 0.0f;
#pragma unroll 1
                        for (int p0 = 0; p0 < DIMP / 4; p0 += PL) {
                            float c[PC][4]; // (beyond dim: zeros on both sides, which change no sum of squares)
#pragma unroll
                            for (int i = 0; i < PC; ++i) {
                                const int j = (tid + i * NT) / PL;
                                load4(c[i], book + (size_t)j * dim, p0 + tid % PL, dim, vec, j < k);
                            }
#pragma unroll
                            for (int i = 0; i < PC; ++i) {
                                const int j = (tid + i * NT) / PL, p = tid % PL;
                                if (PL * BN >= NT || j < BN) planes[p * BN + (j ^ p)] = make_float4(c[i][0], c[i][1], c[i][2], c[i][3]);
                            }
                            __syncthreads();
                            if (here > 0 && lo < k) {
#pragma unroll 1
                                for (int p = 0; p < PL; ++p) {
                                    const float4 c0 = planes[p * BN + ((lo + lane) ^ p)], c1 = planes[p * BN + ((lo + 32 + lane) ^ p)];
                                    const float4 *xp = rows + at * (DIMP / 4) + p0 + p;
#pragma unroll
                                    for (int g0 = 0; g0 < PASS_ROWS; g0 += 4) { // (beyond the last row: what lies there, to no effect)
                                        if (g0 >= here) break;
                                        float4 x4[4];
#pragma unroll
                                        for (int g = 0; g < 4; ++g) x4[g] = xp[(g0 + g) * (DIMP / 4)];
#pragma unroll
                                        for (int g = 0; g < 4; ++g) square_differences(d[0][g0 + g], x4[g], c0), square_differences(d[1][g0 + g], x4[g], c1);
                                    }
                                }
                            }
                            __syncthreads();
                        }
#pragma unroll
                        for (int g = 0; g < PASS_ROWS; ++g) {
                            if (g >= here || lo >= k) break;
                            const int pos = pass + at + g;
                            const uint32_t *mask = &sh.mask[sh.open[pos]][lo >> 5];
                            uint32_t u = 0xFFFFFFFFu, j = 0u;
                            bool stuck = false; // the reference's scan starts at centroid 0: a NaN there stays
#pragma unroll
                            for (int half = 0; half < 2; ++half) {
                                const float dist = P.euclid ? __fsqrt_rn(d[half][g]) : d[half][g];
                                if (!(mask[half] >> lane & 1u)) continue;
                                if (dist < VQB_DENSE_INF && __float_as_uint(dist) < u) u = __float_as_uint(dist), j = lo + 32 * half + lane;
                                stuck = stuck || (lo + 32 * half + lane == 0 && !(dist == dist));
                            }
                            stuck = __any_sync(0xffffffffu, stuck);
                            const uint32_t low = __reduce_min_sync(0xffffffffu, u), first_j = __reduce_min_sync(0xffffffffu, u == low ? j : 0xFFFFFFFFu); // of equal ones the first
                            if (lane == 0 && (stuck || low != 0xFFFFFFFFu)) atomicMin(&sh.least[pos], stuck ? 0ull : (unsigned long long)low << 32 | first_j);
                        }
                    }
                    __syncthreads();
                    if (many) code = (int)(uint32_t)sh.least[place];
                }
            }
            if (P.out_codes && sub == 0 && my_row < P.n) P.out_codes[my_row * P.stages + st] = live ? (uint32_t)code : 0xFFFFFFFFu;
            // ---- 5. residual and sum of the rows that take part, all centroids on their way at once
            const int from = live ? code : -1;
            {
                float c[NI][4];
                uint32_t go = 0;
#pragma unroll
                for (int i = 0; i < NI; ++i) {
                    const int j = __shfl_sync(0xffffffffu, from, side * L + i * LPR);
                    go |= (j >= 0 ? 1u : 0u) << i;
                    load4(c[i], book + (size_t)max(j, 0) * dim, piece, dim, vec, true);
                }
#pragma unroll
                for (int i = 0; i < NI; ++i)
                    if (go >> i & 1u) {
#pragma unroll
                        for (int e = 0; e < 4; ++e) v[i][e] = __fsub_rn(v[i][e], c[i][e]), q[i][e] = __fadd_rn(q[i][e], c[i][e]);
                    }
            }
            if (st + 1 < P.stages) {
                // The reference compares the root of the SERIAL sum of squares (src/rvq.rs:204-207), which lies within 2 dim 2^-24 of this
                // one: only a row that close to epsilon is added up in order.
                float a[NI];
#pragma unroll
                for (int i = 0; i < NI; ++i) a[i] = fmaf(v[i][0], v[i][0], fmaf(v[i][1], v[i][1], fmaf(v[i][2], v[i][2], v[i][3] * v[i][3])));
                const float nrm = sqrtf(sum_rows<NI, L>(a, lane)), slack = 1e-4f * P.epsilon;
                bool below = nrm < P.epsilon - slack;
                uint32_t close = __ballot_sync(0xffffffffu, live && !below && !(nrm > P.epsilon + slack) && sub == 0);
                while (close) {
                    const int r = row_of(__ffs(close) - 1);
                    close &= close - 1;
                    float xr[4];
                    pick_row(xr, r);
                    if (lane < DIMP / 4) *scratch(0, lane) = make_float4(__fmul_rn(xr[0], xr[0]), __fmul_rn(xr[1], xr[1]), __fmul_rn(xr[2], xr[2]), __fmul_rn(xr[3], xr[3]));
                    __syncwarp();
                    const float d = serial_sum(0);
                    if (own_row == r) below = __fsqrt_rn(d) < P.epsilon;
                    __syncwarp();
                }
                if (below) live = false;
            }
        }
        if (!ok) break;
        if (P.out_f16) {
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const unsigned long long row = row0 + i * RL + side;
                if (row >= P.n) continue;
                uint16_t *o = P.out_f16 + row * dim + 4 * piece;
                if (vec) {
                    if (4 * piece < dim)
                        *reinterpret_cast<uint2 *>(o) = make_uint2((uint32_t)f32_to_f16_bits(q[i][0]) | ((uint32_t)f32_to_f16_bits(q[i][1]) << 16),
                                                                   (uint32_t)f32_to_f16_bits(q[i][2]) | ((uint32_t)f32_to_f16_bits(q[i][3]) << 16));
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (4 * piece + e < dim) o[e] = f32_to_f16_bits(q[i][e]);
                }
            }
        }
    }
    // (after an abort: a codebook that is still on its way has to land before the CTA goes; a bounded wait, and at once for a phase that is over)
    if (!ok && tid == 0 && loads > 0) mbar_wait(&sh.bars.bfull, (loads - 1) & 1u, abort_flag, P.error, 43);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN) : "memory");
    }
}

template <int THREADS> __global__ void __launch_bounds__(THREADS) rvq_books_kernel(const float *books, int k, int dim, int dimp, int bn, int vec, float *frames, uint16_t *image, float *extra)
{
    __shared__ BookShared<THREADS / 32> sh;
    next_kernel_may_start();
    make_book<THREADS>(sh, books, blockIdx.x, k, dim, dimp, bn, vec != 0, frames, image, extra);
}

// False: a cooperative launch whose CTAs cannot all be resident (SMs that this process may not use)
template <int KS, int BN, int ROWS> bool launch_stages(CudaDevice &dev, const CUtensorMap &map, const RvqStagesParams &p)
{
    auto kernel = rvq_stages_kernel<KS, BN, ROWS>;
    constexpr size_t smem = stages_smem<KS, BN>();
    static std::atomic<unsigned long long> configured{0}; // bit d: the attribute has been set on device d (it is per device and sticky)
    const unsigned long long bit = 1ull << (dev.device() & 63);
    if (!(configured.load(std::memory_order_relaxed) & bit)) {
        VQB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        configured.fetch_or(bit, std::memory_order_relaxed);
    }
    const unsigned grid = (unsigned)std::min<unsigned long long>((p.n + NWARP * ROWS - 1) / (NWARP * ROWS), (unsigned long long)dev.sm_count());
    KernelScope ks(dev, "rvq_quantize");
    if (p.one) {
        void *args[] = {const_cast<CUtensorMap *>(&map), const_cast<RvqStagesParams *>(&p)};
        const cudaError_t e = cudaLaunchCooperativeKernel((const void *)kernel, dim3(grid), dim3(NT), args, smem, dev.stream());
        if (e == cudaErrorCooperativeLaunchTooLarge) {
            cudaGetLastError();
            return false;
        }
        VQB_CUDA_CHECK(e);
    } else launch_following(kernel, grid, NT, smem, dev.stream(), map, p);
    dev.count_launch();
    return true;
}

template <int KS> bool launch_ks(CudaDevice &dev, const CUtensorMap &map, const RvqStagesParams &p, int bn)
{
    const bool few = p.n <= (unsigned long long)dev.sm_count() * (BM / 2);
    if (bn == 256) return few ? launch_stages<KS, 256, 4>(dev, map, p) : launch_stages<KS, 256, 8>(dev, map, p);
    return few ? launch_stages<KS, 128, 4>(dev, map, p) : launch_stages<KS, 128, 8>(dev, map, p);
}

int book_rows(int k) { return k > 128 ? 256 : 128; }

} // namespace

static bool whole_pieces(const GenericParams &g) { return g.sd % 4 == 0 && (reinterpret_cast<uintptr_t>(g.centroids) & 15u) == 0; }

// Against direct.cu (us a call, here / there): a stage takes 3 to 6 us here up to 64 rows per SM whatever the rows, and 17 us come before; there it
// is the rows' time.  The two meet (256 centroids) at 1300 x 128, 2 stages: 29 / 29; 800 x 96, 4: 39 / 39; 700 x 64, 8: 48 / 48;
// 1150 x 32, 8: 43 / 43; 300 x 61, 4 (no whole 16-byte pieces: no TMA there): 33 / 34.  Up to 128 centroids (128-wide, 8 stages) this
// one is ahead from 300 rows on, but with codebooks of many equal centroids, which cost it nothing: not a line to draw for others.
bool rvq_stages_pays(const GenericParams &g)
{
    if (!whole_pieces(g)) return g.n >= 300;
    return (double)g.n >= (500.0 + 1600.0 / g.stages) * (g.sd < 64 ? 1.5 : 1.0);
}

// Up to the rows that direct.cu used to take, the encode stays one launch of one kernel, as callers have it: the first CTAs make the codebooks'
// images and all wait for them.  They wait at the barrier that every cooperative launch has of its own; counters of the context, which an earlier
// form had, were also those of a captured encode that is replayed beside other calls.  (All CTAs of such a launch are resident, and none leaves
// before the barrier.)  4,999 x 128, 8 stages: 67 us (63 in two launches); beyond, where there were several launches a stage, it is two, and no CTA
// waits for another.
bool rvq_stages_one_launch(const GenericParams &g)
{
    const double rows = (g.k > 128 ? 2.0e6 : g.k > 64 ? 4.6e6 : 6.8e6) / (double)(dense_padded(g.sd) + 32);
    return (double)g.n <= rows * (whole_pieces(g) ? 1.0 : 0.6);
}

size_t rvq_stages_bytes(size_t dim, size_t k, size_t stages)
{
    const size_t bn = book_rows((int)k);
    return stages * (bn * (4 * dense_padded(dim) + 32) + F_FLOATS * sizeof(float));
}

void launch_rvq_stages(CudaDevice &dev, const GenericParams &g, bool euclid, void *work)
{
    const int dimp = (int)dense_padded(g.sd), bn = book_rows(g.k);
    const size_t rows = (size_t)g.stages * bn;
    uint16_t *image = static_cast<uint16_t *>(work); // (whole multiples of 16 bytes follow each other)
    float *extra = reinterpret_cast<float *>(image + rows * 2 * dimp), *frames = extra + rows * 8;
    const bool whole = whole_pieces(g);
    const bool one = rvq_stages_one_launch(g);
    auto make_books = [&] {
        KernelScope ks(dev, "rvq_books");
        rvq_books_kernel<1024><<<g.stages, 1024, 0, dev.stream()>>>(g.centroids, g.k, g.sd, dimp, bn, whole, frames, image, extra);
        VQB_CUDA_CHECK(cudaGetLastError());
        dev.count_launch();
    };
    if (!one) make_books();
    const CUtensorMap map = make_tensor_map_2d(image, 2 * (unsigned long long)dimp, rows, CHUNK, (unsigned)bn, CU_TENSOR_MAP_SWIZZLE_128B);
    RvqStagesParams p = {};
    p.x = g.x, p.books = g.centroids, p.n = g.n, p.dim = g.sd, p.k = g.k, p.stages = g.stages, p.euclid = euclid, p.epsilon = g.epsilon;
    p.vec = whole && (reinterpret_cast<uintptr_t>(g.x) & 15u) == 0 && (reinterpret_cast<uintptr_t>(g.out_f16) & 7u) == 0;
    p.frames = frames, p.image = image, p.extra = extra, p.book_vec = whole, p.one = one, p.out_f16 = g.out_f16, p.out_codes = g.out_codes, p.error = dev.error_word();
    auto launch = [&] {
        switch (dimp / 16) {
        case 2: return launch_ks<2>(dev, map, p, bn);
        case 3: return launch_ks<3>(dev, map, p, bn);
        case 4: return launch_ks<4>(dev, map, p, bn);
        case 5: return launch_ks<5>(dev, map, p, bn);
        case 6: return launch_ks<6>(dev, map, p, bn);
        case 7: return launch_ks<7>(dev, map, p, bn);
        default: return launch_ks<8>(dev, map, p, bn);
        }
    };
    if (!launch()) {
        make_books();
        p.one = 0;
        launch();
    }
}

} // namespace vqb
