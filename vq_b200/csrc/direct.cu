// direct.cu -- nearest centroids of few rows in ONE launch: product-quantizer encode (src/pq.rs:146-187, src/opq.rs:235-264) and
// the residual encoder with all its stages (src/rvq.rs:171-215).
//
// The kernels for large batches need thousands of rows to pay for what they do first (operand tiles, tensor memory, whole
// codebooks in every CTA) or run in several launches per stage; a request with one vector or a few hundred only waits for
// that.  Here a CTA takes a handful of rows, and its threads share out the CENTROIDS: thread t owns centroids t and t + TK.
// The codebook streams through a ring of shared-memory chunks (up to 16 dimensions of all centroids each, two to five chunks
// ahead), across the stages of a residual encode without a break, since the order of the chunks does not depend on the
// choices.  Wide codebooks come by TMA (one thread, one instruction a chunk: 16-byte cp.async by all threads spent 490 cycles
// on a chunk that takes 700 to use), narrow or unaligned ones by cp.async.
//
// Euclidean metrics rank with S_j = |c_j|^2/2 - x.c_j (one FMA per dimension instead of the reference's three rounded
// operations) and accept the smallest S when every other one is farther away than the margin below; otherwise the
// centroids within the margin are evaluated with the reference's arithmetic.  Other metrics are evaluated exactly at once.
//
// Margin.  u = 2^-24, d dimensions (padded to whole chunks), xh = |x|^2/2, HN = max_j |c_j|^2/2, L = d/2 + 4: the products of even
// and odd dimensions are added up side by side (packed FMAs), so no term passes through more than L roundings.
//   |S_j - true| <= E = L u (xh + 3 HN)     (sum |x_i c_ji| <= xh + hn_j; hn_j added up the same way; one subtraction)
//   the reference's own chain of d terms and, for Euclidean, sqrt: it can prefer w over a only if D_w <= D_a (1 + 2.02 (d + 4)u),
//   D_a = 2 (xh + S_a)   =>   S_w - S_a <= 2E + 2.1 (d + 5)u (xh + S_a)
// (xh + S_a cancels; 1e-3 (xh + HN) covers its rounding), plus 1e-36 for products that underflow; rows with xh + HN >= 1e37
// (or NaN) are evaluated exactly as a whole.
#include <algorithm>
#include <atomic>
#include <cstring>

#include "assign_filter.cuh"
#include "cuda_device.hpp"
#include "direct.cuh"
#include "kernels_common.cuh"
#include "tma_host.hpp"
#include "umma.cuh"

namespace vqb {

namespace {

constexpr int DT = 256;  // threads of a CTA: DT / TK groups of TK threads, each group with its own R rows
constexpr int DC = 16;   // dimensions of a codebook chunk
constexpr int DK_MAX = 256;
constexpr size_t STATIC_SMEM = 8192; // more than the kernels' own shared arrays, which count towards the 48 KiB of a launch that asks for no more

struct DirectParams {
    const float *x;
    unsigned long long n, ld;
    int m, k, sd, tk;       // tk: threads per group, 32, 64 or 128; 2 tk >= k
    const float *centroids; // [m][k][sd], or [stages][k][sd]
    uint16_t *out_f16;
    uint32_t *out_codes;
    float *out_f32;
    float pv, epsilon;
    int stages;             // 0: product-quantizer encode, gridDim.y sub-spaces
    int vec4;               // centroids are whole 16-byte pieces
    int tma;                // chunks of 16 dimensions come by TMA
    int *error;             // set when a bounded wait expires
};

template <int BYTES> __device__ __forceinline__ void cp_async_zfill(uint32_t dst, const float *src, bool in)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(dst), "l"(src), "n"(BYTES), "r"(in ? BYTES : 0) : "memory");
}

// unsigned order of the bits = order of the floats (not for NaN)
__device__ __forceinline__ uint32_t ordered_bits(float v)
{
    const uint32_t b = __float_as_uint(v);
    return b ^ ((b >> 31) ? 0xFFFFFFFFu : 0x80000000u);
}
__device__ __forceinline__ float from_ordered_bits(uint32_t u) { return __uint_as_float(u ^ ((u >> 31) ? 0x80000000u : 0xFFFFFFFFu)); }

// A chunk row holds dc = 4, 8 or 16 floats = 1, 2 or 4 pieces of 16 bytes, permuted by the row's number, so that eight lanes read
// the same piece of eight rows without a bank conflict.
__host__ __device__ __forceinline__ int chunk_dims(int sd) { return sd <= 4 ? 4 : sd <= 8 ? 8 : DC; }
// (For 16 dimensions this is the TMA's 64-byte swizzle.)
__device__ __forceinline__ int chunk_swizzle(int dc, int row) { return dc == 16 ? (row >> 1) & 3 : dc == 8 ? (row >> 2) & 1 : 0; }
// chunks in the ring: with one row per group there is about one CTA per SM and its time is the way to memory
__host__ __device__ constexpr int ring_depth(int r) { return r == 1 ? 6 : 3; }

template <int METRIC, int R> __global__ void __launch_bounds__(DT, 3) direct_kernel(const __grid_constant__ CUtensorMap books, const DirectParams P)
{
    constexpr bool FILTER = METRIC == M_SQ || METRIC == M_EUCLID;
    constexpr int NBUF = ring_depth(R), NW = DT / 32;
    extern __shared__ __align__(1024) float smem[];
    const int k = P.k, sd = P.sd, tk = P.tk, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int groups = DT / tk, rows = groups * R;          // rows of this CTA
    const int g = tid / tk, t = tid % tk;                   // group, place in it
    const int dc = chunk_dims(sd);
    const int nch = (sd + dc - 1) / dc, xstr = nch * dc;    // rows are padded with zeros to whole chunks
    const bool rvq = P.stages > 0;
    const int s = blockIdx.y, nst = rvq ? P.stages : 1;
    float *ring = smem;                                     // [NBUF][2 tk][dc]
    const int chunk_floats = 2 * tk * dc;
    float *xs = ring + NBUF * chunk_floats;                 // [rows][xstr]
    float *qs = xs + rows * xstr;                           // [rows][xstr], residual encoder only
    __shared__ float s_sq[NW * R];                          // sum of squares of a row, serial
    __shared__ float s_min[NW][R];
    __shared__ float s_hn[NW];
    __shared__ uint32_t s_mask[NW * R][DK_MAX / 32];        // FILTER: the candidates of a row
    __shared__ uint8_t s_list[FILTER ? NW : 1][DK_MAX];     // and, per warp, their numbers
    __shared__ unsigned long long s_key[NW * R];            // other metrics: (distance, centroid)
    __shared__ int s_code[NW * R];
    __shared__ uint8_t s_done[NW * R];
    __shared__ unsigned long long s_full[NBUF];             // TMA: a chunk has arrived
    __shared__ int s_abort;

    const unsigned long long row0 = (unsigned long long)blockIdx.x * rows;
    const int have = (int)min((unsigned long long)rows, P.n - row0);

    // ---- the codebook ring ------------------------------------------------------------------------------------------
    // Thread's place in a chunk: piece lcol of the rows lrow, lrow + lstep, ... (16 bytes each, or 4).  lstep is a multiple of 16,
    // so the permutation is the same for all of them.
    const int lpieces = P.vec4 ? dc / 4 : dc, lrow = tid / lpieces, lcol = tid % lpieces, lstep = DT / lpieces;
    const int ld0 = P.vec4 ? 4 * lcol : lcol; // first of its dimensions
    const uint32_t ldst = (uint32_t)__cvta_generic_to_shared(ring) + 4u * (lrow * dc + (ld0 ^ (4 * chunk_swizzle(dc, lrow))));
    int lst = 0, lch = 0, lslot = 0; // stage, chunk and ring slot of the next load
    auto load_chunk = [&] {
        if (P.tma) {
            if (tid == 0 && lst < nst) {
                mbar_expect_tx(&s_full[lslot], 4u * chunk_floats);
                tma_load_2d(ring + lslot * chunk_floats, &books, lch * DC, (rvq ? lst : s) * k, &s_full[lslot]);
                if (++lch == nch) lch = 0, ++lst;
                if (++lslot == NBUF) lslot = 0;
            }
            return;
        }
        if (lst < nst) {
            const int d = lch * dc + ld0;
            const float *src = P.centroids + (size_t)(rvq ? lst : s) * k * sd + (size_t)lrow * sd + d;
            uint32_t dst = ldst + 4u * lslot * chunk_floats;
            for (int row = lrow; row < 2 * tk; row += lstep) {
                const bool in = row < k && d < sd;
                if (P.vec4) cp_async_zfill<16>(dst, in ? src : P.centroids, in);
                else cp_async_zfill<4>(dst, in ? src : P.centroids, in);
                src += (size_t)lstep * sd, dst += 4u * lstep * dc;
            }
            if (++lch == nch) lch = 0, ++lst;
            if (++lslot == NBUF) lslot = 0;
        }
        asm volatile("cp.async.commit_group;" ::: "memory"); // also when empty: the number of pending groups stays fixed
    };
    if (P.tma) {
        if (tid == 0) {
            for (int b = 0; b < NBUF; ++b) mbar_init(&s_full[b], 1);
            s_abort = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        __syncthreads();
    }
    for (int q = 0; q < NBUF - 1; ++q) load_chunk();

    // ---- the rows ---------------------------------------------------------------------------------------------------
    for (int r = warp; r < rows; r += NW) {
        for (int i = lane; i < xstr; i += 32) {
            xs[r * xstr + i] = (r < have && i < sd) ? __ldg(P.x + (row0 + r) * P.ld + (size_t)s * sd + i) : 0.0f;
            if (rvq) qs[r * xstr + i] = 0.0f;
        }
    }
    if (tid < rows) s_done[tid] = tid < have ? 0 : 1;
    __syncthreads();
    auto square_sums = [&] { // serial per row: also the residual's norm and the cosine's
        if (tid < rows) {
            const float *xr = xs + tid * xstr;
            float a = 0.0f;
#pragma unroll 4
            for (int i = 0; i < xstr; i += 4) { // the padding adds +0 to a sum of squares
                const float4 v = *reinterpret_cast<const float4 *>(xr + i);
                a = __fadd_rn(a, __fmul_rn(v.x, v.x)), a = __fadd_rn(a, __fmul_rn(v.y, v.y));
                a = __fadd_rn(a, __fmul_rn(v.z, v.z)), a = __fadd_rn(a, __fmul_rn(v.w, v.w));
            }
            s_sq[tid] = a;
        }
    };
    if (FILTER || METRIC == M_COSINE) square_sums();

    const int ja = t, jb = t + tk;
    const int swa = 4 * chunk_swizzle(dc, ja), swb = 4 * chunk_swizzle(dc, jb);
    const float *xg = xs + g * R * xstr;
    int slot = 0;
    uint32_t phase = 0;
    for (int st = 0; st < nst; ++st) {
        const float *cbk = P.centroids + (size_t)(rvq ? st : s) * k * sd;
        if (!FILTER && tid < rows) s_key[tid] = ~0ull;
        // FILTER: pairs of partial sums of x.c and |c|^2; else DistAcc's sums and the centroids' squares
        f32x2 p0[R], p1[R], m0 = 0ull, m1 = 0ull;
        float a0[R], a1[R], n0 = 0.0f, n1 = 0.0f;
#pragma unroll
        for (int r = 0; r < R; ++r) a0[r] = a1[r] = 0.0f, p0[r] = p1[r] = 0ull;
        for (int ch = 0; ch < nch; ++ch) {
            if (P.tma) mbar_wait<200u>(&s_full[slot], phase, &s_abort, P.error, 21);
            else asm volatile("cp.async.wait_group %0;" ::"n"(NBUF - 2) : "memory");
            __syncthreads(); // this chunk is there for everybody, and the one before is used up
            load_chunk();
            const float *c = ring + slot * chunk_floats;
            if (++slot == NBUF) slot = 0, phase ^= 1u;
            const float *ca = c + ja * dc, *cb = c + jb * dc, *xc = xg + ch * dc;
            auto four = [&](int i) { // four dimensions
                if (FILTER) {
                    const ulonglong2 va = *reinterpret_cast<const ulonglong2 *>(ca + (i ^ swa)), vb = *reinterpret_cast<const ulonglong2 *>(cb + (i ^ swb));
                    m0 = fma2(va.x, va.x, m0), m1 = fma2(vb.x, vb.x, m1);
                    m0 = fma2(va.y, va.y, m0), m1 = fma2(vb.y, vb.y, m1);
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const ulonglong2 xv = *reinterpret_cast<const ulonglong2 *>(xc + r * xstr + i);
                        p0[r] = fma2(xv.x, va.x, p0[r]), p1[r] = fma2(xv.x, vb.x, p1[r]);
                        p0[r] = fma2(xv.y, va.y, p0[r]), p1[r] = fma2(xv.y, vb.y, p1[r]);
                    }
                } else {
                    const float4 ca4 = *reinterpret_cast<const float4 *>(ca + (i ^ swa)), cb4 = *reinterpret_cast<const float4 *>(cb + (i ^ swb));
                    const float va[4] = {ca4.x, ca4.y, ca4.z, ca4.w}, vb[4] = {cb4.x, cb4.y, cb4.z, cb4.w};
                    if (METRIC == M_COSINE) {
#pragma unroll
                        for (int u = 0; u < 4; ++u) n0 = __fadd_rn(n0, __fmul_rn(va[u], va[u])), n1 = __fadd_rn(n1, __fmul_rn(vb[u], vb[u]));
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const float4 x4 = *reinterpret_cast<const float4 *>(xc + r * xstr + i);
                        const float xv[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            if (METRIC == M_COSINE) {
                                a0[r] = __fadd_rn(a0[r], __fmul_rn(xv[u], va[u])), a1[r] = __fadd_rn(a1[r], __fmul_rn(xv[u], vb[u]));
                            } else {
                                DistAcc<METRIC> acc;
                                acc.a = a0[r], acc.step(xv[u], va[u], P.pv), a0[r] = acc.a;
                                acc.a = a1[r], acc.step(xv[u], vb[u], P.pv), a1[r] = acc.a;
                            }
                        }
                    }
                }
            };
            if (dc == DC && METRIC != M_MINKOWSKI) {
#pragma unroll
                for (int i = 0; i < DC; i += 4) four(i);
            } else {
#pragma unroll 1
                for (int i = 0; i < dc; i += 4) four(i);
            }
        }
        // ---- the smallest of a row over the threads of its group ----------------------------------------------------
        if (FILTER) {
            n0 = 0.5f * hsum2(m0), n1 = 0.5f * hsum2(m1);
            const float hn = __uint_as_float(__reduce_max_sync(0xffffffffu, max(ja < k ? __float_as_uint(fmaxf(n0, 0.0f)) : 0u,
                                                                                 jb < k ? __float_as_uint(fmaxf(n1, 0.0f)) : 0u)));
            if (lane == 0) s_hn[warp] = hn;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                a0[r] = ja < k ? n0 - hsum2(p0[r]) : VQB_INF;
                a1[r] = jb < k ? n1 - hsum2(p1[r]) : VQB_INF;
                const uint32_t u = __reduce_min_sync(0xffffffffu, ordered_bits(fminf(fminf(a0[r], a1[r]), VQB_INF)));
                if (lane == 0) s_min[warp][r] = from_ordered_bits(u);
            }
            __syncthreads();
            float hmax = 0.0f;
#pragma unroll
            for (int w = 0; w < NW; ++w) hmax = fmaxf(hmax, s_hn[w]); // all groups look at the same centroids
            const float u24 = 5.9604645e-8f, e2 = 2.0f * (float)(xstr / 2 + 4) * u24, own = 2.1f * (float)(sd + 5) * u24;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float best = s_min[g * (tk / 32)][r];
                for (int w = 1; w < tk / 32; ++w) best = fminf(best, s_min[g * (tk / 32) + w][r]);
                const float xh = 0.5f * s_sq[g * R + r];
                const float limit = xh + hmax < 1e37f ? best + (e2 * (xh + 3.0f * hmax) + own * (fmaxf(xh + best, 0.0f) + 1e-3f * (xh + hmax)) + 1e-36f)
                                                      : VQB_INF; // also for NaN: everything is a candidate
                const unsigned b0 = __ballot_sync(0xffffffffu, ja < k && !(a0[r] > limit)), b1 = __ballot_sync(0xffffffffu, jb < k && !(a1[r] > limit));
                if (lane == 0) s_mask[g * R + r][t >> 5] = b0, s_mask[g * R + r][(t + tk) >> 5] = b1;
            }
            __syncthreads();
            // A row with one candidate has its answer.  The others' candidates are evaluated in the reference's arithmetic, a row
            // per warp and a candidate per lane (dead clusters leave dozens of equal centroids behind), lowest index of the
            // smallest distance.
            for (int r = warp; r < have; r += NW) {
                int cnt = 0;
                for (int w = 0; w < tk / 16; ++w) {
                    const uint32_t word = s_mask[r][w];
                    if (word >> lane & 1u) s_list[warp][cnt + __popc(word & ((1u << lane) - 1u))] = (uint8_t)(w * 32 + lane);
                    cnt += __popc(word);
                }
                __syncwarp();
                if (cnt == 1) {
                    if (lane == 0) s_code[r] = s_list[warp][0];
                } else {
                    uint32_t best = 0xFFFFFFFFu;
                    int code = 0; // stays where nothing is below +inf
                    bool stuck = false;
                    for (int base = 0; base < cnt; base += 32) {
                        const bool in = base + lane < cnt;
                        const int j = s_list[warp][in ? base + lane : 0];
                        const float *xr = xs + r * xstr, *c = cbk + (size_t)j * sd;
                        float d = 0.0f;
                        auto add = [&](float xv, float cv) {
                            const float e = __fsub_rn(xv, cv);
                            d = __fadd_rn(d, __fmul_rn(e, e));
                        };
                        if (P.vec4) {
#pragma unroll 16
                            for (int i = 0; i < sd; i += 4) {
                                const float4 cv = __ldg(reinterpret_cast<const float4 *>(c + i)), xv = *reinterpret_cast<const float4 *>(xr + i);
                                add(xv.x, cv.x), add(xv.y, cv.y), add(xv.z, cv.z), add(xv.w, cv.w);
                            }
                        } else {
#pragma unroll 16
                            for (int i = 0; i < sd; ++i) add(xr[i], __ldg(c + i));
                        }
                        if (METRIC == M_EUCLID) d = __fsqrt_rn(d);
                        stuck = stuck || __any_sync(0xffffffffu, in && j == 0 && !(d == d)); // the scan starts at centroid 0: a NaN there stays
                        const uint32_t u = in && d < VQB_INF ? ordered_bits(d) : 0xFFFFFFFFu, um = __reduce_min_sync(0xffffffffu, u);
                        const int jm = (int)__reduce_min_sync(0xffffffffu, u == um ? (unsigned)j : 0xFFFFFFFFu);
                        if (um < best) best = um, code = jm;
                    }
                    if (lane == 0) s_code[r] = stuck ? 0 : code;
                }
                __syncwarp();
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                DistAcc<METRIC> acc;
                const float na = METRIC == M_COSINE ? __fsqrt_rn(s_sq[g * R + r]) : 0.0f;
                acc.a = a0[r], acc.b = n0;
                const float d0 = acc.finish(P.pv, na);
                acc.a = a1[r], acc.b = n1;
                const float d1 = acc.finish(P.pv, na);
                const uint32_t u0 = ja < k && d0 < VQB_INF ? ordered_bits(d0) : 0xFFFFFFFFu, u1 = jb < k && d1 < VQB_INF ? ordered_bits(d1) : 0xFFFFFFFFu;
                const uint32_t um = __reduce_min_sync(0xffffffffu, min(u0, u1));
                const uint32_t jm = __reduce_min_sync(0xffffffffu, u0 == um ? (uint32_t)ja : u1 == um ? (uint32_t)jb : 0xFFFFFFFFu);
                if (lane == 0 && um != 0xFFFFFFFFu) atomicMin(s_key + g * R + r, ((unsigned long long)um << 32) | jm);
                if (ja == 0 && !(d0 == d0)) atomicMin(s_key + g * R + r, 0ull);
            }
            __syncthreads();
            // The reference's scan starts at centroid 0 and replaces it on strict '<' only: a NaN there (key 0) stays, and
            // nothing below +inf (key untouched) leaves it in place too.
            if (tid < rows) s_code[tid] = s_key[tid] == ~0ull ? 0 : (int)(uint32_t)s_key[tid];
        }
        __syncthreads();
        if (!rvq) break;
        // ---- residual and running sum of the rows that still go on -----------------------------------------------------
        // (two rows and up to four pieces of them per warp at a time: the loads of a turn are on their way together)
        for (int r0 = warp; r0 < have; r0 += 2 * NW) {
            for (int i0 = lane; i0 < sd; i0 += 128) {
                float v[2][4];
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int r = r0 + h * NW, i = i0 + 32 * u;
                        v[h][u] = r < have && i < sd ? __ldg(cbk + (size_t)s_code[r] * sd + i) : 0.0f;
                    }
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int r = r0 + h * NW, i = i0 + 32 * u;
                        if (r < have && i < sd && !s_done[r]) {
                            xs[r * xstr + i] = __fsub_rn(xs[r * xstr + i], v[h][u]);
                            qs[r * xstr + i] = __fadd_rn(qs[r * xstr + i], v[h][u]);
                        }
                    }
            }
        }
        __syncthreads();
        square_sums();
        if (tid < have) {
            if (P.out_codes) P.out_codes[(row0 + tid) * P.stages + st] = s_done[tid] ? 0xFFFFFFFFu : (uint32_t)s_code[tid];
            if (__fsqrt_rn(s_sq[tid]) < P.epsilon) s_done[tid] = 1;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");

    // ---- results ------------------------------------------------------------------------------------------------------
    if (rvq) {
        __syncthreads();
        if (P.out_f16)
            for (int r = warp; r < have; r += NW)
                for (int i = lane; i < sd; i += 32) P.out_f16[(row0 + r) * sd + i] = f32_to_f16_bits(qs[r * xstr + i]);
    } else {
        const size_t dim = (size_t)P.m * sd;
        const float *cbk = P.centroids + (size_t)s * k * sd;
        for (int e = tid; e < have * sd; e += DT) {
            const int r = e / sd, i = e % sd;
            const float v = __ldg(cbk + (size_t)s_code[r] * sd + i);
            const size_t at = (row0 + r) * dim + (size_t)s * sd + i;
            if (P.out_f16) P.out_f16[at] = f32_to_f16_bits(v);
            if (P.out_f32) P.out_f32[at] = v;
        }
        if (P.out_codes && tid < have) P.out_codes[(row0 + tid) * P.m + s] = (uint32_t)s_code[tid];
    }
}

} // namespace

static size_t direct_smem(int r, int tk, int sd, bool rvq)
{
    const int dc = chunk_dims(sd), xstr = (sd + dc - 1) / dc * dc, rows = DT / tk * r;
    return sizeof(float) * ((size_t)ring_depth(r) * 2 * tk * dc + (size_t)rows * xstr * (rvq ? 2 : 1));
}

static int direct_tk(int k) { return k > 128 ? 128 : k > 64 ? 64 : 32; }

// Rows per thread group.  A CTA's time is about its rows plus what it does once (3 rows' worth: the codebook through the ring,
// barriers), and the SM with the most CTAs sets the kernel's.
static int direct_rows(unsigned long long n, int m, int tk, int sm_count)
{
    int best = 1;
    unsigned long long least = ~0ull;
    for (int r : {8, 6, 4, 2, 1}) {
        const unsigned long long per = (unsigned long long)(DT / tk) * r, ctas = (n + per - 1) / per * m;
        const unsigned long long cost = (ctas + sm_count - 1) / sm_count * (r + 3);
        if (cost < least) least = cost, best = r;
    }
    return best;
}

template <int METRIC, int R> static void launch_rows(CudaDevice &dev, const CUtensorMap &books, const DirectParams &p, int m)
{
    auto kernel = direct_kernel<METRIC, R>;
    const int rows = DT / p.tk * R;
    const size_t smem = direct_smem(R, p.tk, p.sd, p.stages > 0);
    static std::atomic<unsigned long long> configured{0}; // bit d: the attribute has been set on device d (it is per device and sticky)
    const unsigned long long bit = 1ull << (dev.device() & 63);
    if (smem + STATIC_SMEM > 48 * 1024 && !(configured.load(std::memory_order_relaxed) & bit)) {
        VQB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(dev.smem_limit() - STATIC_SMEM)));
        configured.fetch_or(bit, std::memory_order_relaxed);
    }
    KernelScope ks(dev, p.stages > 0 ? "rvq_quantize" : "pq_encode");
    kernel<<<dim3((unsigned)((p.n + rows - 1) / rows), m), DT, smem, dev.stream()>>>(books, p);
    VQB_CUDA_CHECK(cudaGetLastError());
    dev.count_launch();
}

template <int METRIC> static void launch_metric(CudaDevice &dev, DirectParams &p, int m)
{
    CUtensorMap books;
    p.tma = p.vec4 && p.sd > DC / 2 && dev.error_word() != nullptr;
    if (p.tma)
        books = make_tensor_map_2d(p.centroids, p.sd, (unsigned long long)p.k * (p.stages > 0 ? p.stages : m), DC, 2 * p.tk, CU_TENSOR_MAP_SWIZZLE_64B);
    else std::memset(&books, 0, sizeof books);
    p.error = dev.error_word();
    switch (direct_rows(p.n, m, p.tk, dev.sm_count())) {
    case 8: launch_rows<METRIC, 8>(dev, books, p, m); break;
    case 6: launch_rows<METRIC, 6>(dev, books, p, m); break;
    case 4: launch_rows<METRIC, 4>(dev, books, p, m); break;
    case 2: launch_rows<METRIC, 2>(dev, books, p, m); break;
    default: launch_rows<METRIC, 1>(dev, books, p, m); break;
    }
}

static void launch_any(CudaDevice &dev, DirectParams &p, int metric, int m)
{
    switch (metric) {
    case M_SQ: launch_metric<M_SQ>(dev, p, m); break;
    case M_EUCLID: launch_metric<M_EUCLID>(dev, p, m); break;
    case M_COSINE: launch_metric<M_COSINE>(dev, p, m); break;
    case M_MANHATTAN: launch_metric<M_MANHATTAN>(dev, p, m); break;
    case M_CHEBYSHEV: launch_metric<M_CHEBYSHEV>(dev, p, m); break;
    case M_MINKOWSKI: launch_metric<M_MINKOWSKI>(dev, p, m); break;
    case M_HAMMING: launch_metric<M_HAMMING>(dev, p, m); break;
    default: throw Error(90, "unknown metric");
    }
}

// Where the other kernels take over.  A thread looks at two centroids whatever k is, so this kernel's time follows (row, sub-space)
// pairs and 2 tk = 64, 128 or 256.  Measured with rows on the GPU, from the call to its result and as one of many in a row (the
// two agree within a few per cent):
// These lines are of the kernels on the other side before launches overlapped and the tensor-core one became what it is (3000 x 128 now takes
// 15.5 us there, in three launches), and before sub-spaces of 4 values and odd numbers of them went to it as well: they have not been
// drawn anew since, and could lie lower.
//   the tensor-core kernel (8-wide sub-spaces; 19 us in three launches as one of many, hardly dependent on the rows) passes at
//       k 256: 10,900 .. 11,100 pairs (m 4, 8, 16, 32), k 200: 10,750, k 128: 15,900 .. 20,000, k 20, 40, 64: 27,100 .. 27,400
//   the CUDA-core kernels (19 us up to k 20, 33 at 64, 40 .. 46 at 128, 66 .. 83 at 256, until their grids are full, some thousand
//       rows later) pass at  k 256: 57,800 .. 64,400 pairs (4- and 16-wide), 68,600 (8-wide), 78,900 (Manhattan), k 128: 67,000,
//       k 64: 63,700 (cosine), 70,000 (24-wide), k 48: 48,000, k 40: 28,000 (cosine), k 32: 32,000, k 2 .. 20: 16,000 (16-wide) .. 30,000,
//       and k 100 of 5 values, which are no whole 16-byte pieces: 29,000
static bool whole_pieces(int sd, const float *centroids) { return sd % 4 == 0 && (reinterpret_cast<uintptr_t>(centroids) & 15u) == 0; }

bool direct_encode_applicable(const AssignParams &p, bool tensor)
{
    if (p.k > DK_MAX || p.sd > 256 || p.m > 65535) return false;
    const double pairs = (double)p.n * p.m;
    if (tensor) return pairs * (2 * direct_tk(p.k) + 68) <= 3.56e6;
    return pairs <= (p.k < 48 ? 20e3 : 56e3) * (whole_pieces(p.sd, p.centroids) ? 1.0 : 0.5);
}

void launch_direct_encode(CudaDevice &dev, const AssignParams &a, int metric)
{
    DirectParams p = {};
    p.x = a.x, p.n = a.n, p.ld = a.ld, p.m = a.m, p.k = a.k, p.sd = a.sd, p.tk = direct_tk(a.k);
    p.centroids = a.centroids;
    p.out_f16 = a.out_f16, p.out_codes = a.out_codes, p.out_f32 = a.out_f32, p.pv = a.pv;
    p.vec4 = whole_pieces(a.sd, a.centroids);
    launch_any(dev, p, metric, a.m);
}

// Against the CUDA-core kernel this one is ahead at every size that was measured (Manhattan, 80,000 x 128, k 256, 8 stages:
// 7.2 -> 2.8 ms; cosine: 10.1 -> 2.4 ms).  Where the tensor-core kernel takes over: rvq_stages_pays (rvq_tc.cu).
bool direct_rvq_applicable(const GenericParams &g, size_t smem_limit)
{
    return g.k <= DK_MAX && std::max(direct_smem(8, direct_tk(g.k), g.sd, true), direct_smem(1, direct_tk(g.k), g.sd, true)) <= smem_limit - STATIC_SMEM;
}

void launch_direct_rvq(CudaDevice &dev, const GenericParams &g, int metric)
{
    DirectParams p = {};
    p.x = g.x, p.n = g.n, p.ld = g.ld, p.m = 1, p.k = g.k, p.sd = g.sd, p.tk = direct_tk(g.k);
    p.centroids = g.centroids;
    p.out_f16 = g.out_f16, p.out_codes = g.out_codes, p.pv = g.pv, p.epsilon = g.epsilon, p.stages = g.stages;
    p.vec4 = whole_pieces(g.sd, g.centroids);
    launch_any(dev, p, metric, 1);
}

} // namespace vqb
