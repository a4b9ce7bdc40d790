// dense_tc.cu -- full-width nearest-centroid search on the 5th-generation tensor cores (tcgen05 + TMEM + TMA).
//
// The residual quantizer's k-means and encode (src/rvq.rs:107,111-128,186-202) compare every row with every centroid
// over the full dimension: a dense n x k x dim contraction.  This file ranks centroids with
//        S_j = |c_j|^2/2 - x.c_j          (|x - c_j|^2 = |x|^2 + 2 S_j)
// where the dot products come from tcgen05.mma (binary16 inputs, f32 accumulation in tensor memory), keeps for every row
// the SHORTLIST of centroids whose S lies within a proven error bound of the smallest one, decides the rows with a single
// candidate and hands the others to a resolve kernel (resolve.cu) that evaluates only their candidates with the reference's
// exact f32 arithmetic.  The final choice is therefore the reference's; the tensor cores only prune.
//
// Operands.  Rows and centroids move into a common frame, v = s (x - mu): distances scale by s, while |x||c|, which the error
// bound grows with, loses the rows' common part.  mu is about the mean and s about the inverse size of a sample of 256 rows
// (dense_frame_kernel; any values are correct).  v is split into two binary16 numbers, v = h + l + e (the "image" of a row: as many
// bytes as the row itself), and three products are added up: h.ch + h.cl + l.ch.  With one TF32 product (bound 2.1e-3 |x||c|)
// between 15 and 94 % of the rows of a Gaussian mixture went to the exact kernel, which then took 0.31 ms per pass over
// 1M x 128 rows beside 0.13 ms for the shortlist; bf16 instead of binary16 (bound 5.5e-5) still left 50 % in the first stage.
// Three products take 24 MMAs per tile of 128 dimensions and bound the kernel together with the epilogue: 0.148 ms per pass over
// 1M x 128 (0.84 of the measured bf16 rate) beside 0.079 ms of row traffic.  The images are written where the rows are touched
// anyway (dense_prepare_kernel, rvq_apply_kernel); any width up to 128 is padded to whole K steps there.
//
// Bound, in the frame.  |l.cl| + |e.c| + |v.ec| <= 3.01 * 2^-22 sum|v_i c_ji| (l below binary16's normal range: 2^-25 absolute
// instead, <= 2^-25 sqrt(dim) (|v| + |c|)); 25 accumulation steps, each at most 2^-22:
//   |dot_tc - v.c| <= 7e-6 |v| |c_j| + 4e-7 (|v| + |c_j|) =: E
// and with the reference's own chain error (<= (dim + 2) 2^-24 relative on the distance) the winner w satisfies
//   S_w <= S_min + 2 E + 1.05 (dim + 6) 2^-24 (|v|^2 + 2 S_min + 2 E).
// Everything not finite falls out of the comparisons and marks the row for a full exact scan.
//
// Kernel layout (one CTA per SM, persistent over 128-row tiles):
//   warp 0      TMA producer: the codebook's image once (resident in shared memory), then the rows' images in 128-byte
//               column chunks through a 5-stage ring (cp.async.bulk.tensor, 128B swizzle, no multicast)
//   warp 1      allocates tensor memory and issues tcgen05.mma M128 x N256 x K16 (kind::f16); two 256-column
//               accumulators so the next tile's MMAs overlap this tile's epilogue.  One K = 8 step of kind::tf32 per tile multiplies
//               a constant (1, 1, 0, ...) row operand with (-hn_h, -hn_l, 0, ...) per centroid, so the accumulator holds
//               D = x.c - |c|^2/2 = -S and the epilogue never touches the half norms
//   warps 2..5  epilogue: tcgen05.ld the 128 x 256 values, one row per lane; pass 1 finds the largest D and whether it is the only
//               candidate, and which; for a warp with an undecided row pass 2 shifts the sign of (D - limit) into a 256-bit mask
// Every wait is bounded; on expiry the kernel records an error code, stops issuing work and frees its tensor memory.
#include <cuda.h>

#include <algorithm>
#include <mutex>

#include "cuda_device.hpp"
#include "dense_image.cuh"
#include "dense_tc.hpp"
#include "kernels_common.cuh"
#include "tma_host.hpp"
#include "umma.cuh"

namespace vqb {

namespace {

constexpr int BM = 128;          // rows per tile (= TMEM lanes)
constexpr int BN = 256;          // centroids per tile (= accumulator columns)
constexpr int CHUNK = 64;        // binary16 values per 128-byte swizzle row
constexpr int NSTAGE = 5;        // row-tile ring depth (stages of 128 rows x 128 bytes)
constexpr int MAX_KCHUNKS = 4;   // images of up to 2 x 128 values
constexpr uint32_t X_STAGE_BYTES = BM * 128;
constexpr uint32_t C_CHUNK_BYTES = BN * 128;

struct alignas(8) Barriers {
    unsigned long long full[NSTAGE], empty[NSTAGE], cfull, tfull[2], tempty[2];
    uint32_t tmem_base;
    int abort_flag;
};

struct ShortlistParams {
    unsigned long long n;
    int dim, k;
    const float *hn;      // [256] |c_j|^2 / 2 in the frame, +inf beyond k
    const float *frame;
    const float *xnorm2;  // [n]   |v|^2 per row, an upper bound
    uint32_t *cand;       // [n][8] bit j set = centroid j may be the reference's choice (all k bits set: examine all)
    unsigned long long *stats; // [0] rows, [1] candidates, [2] rows needing a full scan   (may be null)
    float *debug_dots;    // [n][256] raw tensor-core dot products (may be null)
    int *error;           // device error word, 0 = ok
    // training passes (codes != null): a row with a single candidate gets its assignment here; the others are appended to
    // `list` (and only they get their mask written)
    uint8_t *codes;        // [n] previous assignment in, new assignment out
    uint32_t *changed;     // VQB_MOVED_BITS is OR-ed in when a row moved (may be null)
    uint32_t *list;        // [n] rows left for the exact decision
    uint32_t *list_count;  // [1] zero on entry
};

// KS: K = 16 steps of one part (h or l) of an image.  A constant, because one thread issues the MMAs: with descriptors worked out
// per step it took 260 cycles an MMA, now 200 with all waits (the tensor core alone: 134).
template <int KS>
__global__ void __launch_bounds__(192, 1) dense_shortlist_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_c,
                                                                const ShortlistParams P)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char *base = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    unsigned char *c_smem = base;                                            // kchunks x 32 KiB
    unsigned char *x_smem = base + (size_t)MAX_KCHUNKS * C_CHUNK_BYTES;       // NSTAGE x 16 KiB
    float *hn_s = reinterpret_cast<float *>(x_smem + (size_t)NSTAGE * X_STAGE_BYTES); // 256 floats (diagnostics only)
    // one more K = 8 step folds the half norms into the accumulator: operand A = (1, 1, 0, ...) for every row, operand B =
    // (-hn_h, -hn_l, 0, ...) per centroid, hn split into two TF32 numbers; both tiles K-major with 32-byte rows, 32B swizzle
    unsigned char *a1_smem = reinterpret_cast<unsigned char *>(hn_s + BN);            // 128 rows x 32 bytes
    unsigned char *bh_smem = a1_smem + BM * 32;                                       // 256 rows x 32 bytes
    Barriers *bars = reinterpret_cast<Barriers *>(bh_smem + BN * 32);
    volatile int *abort_flag = &bars->abort_flag;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned long long n_tiles = (P.n + BM - 1) / BM;
    constexpr int kchunks = (2 * KS + 3) / 4; // 64-element pieces of an image

    if (threadIdx.x == 0) {
        for (int s = 0; s < NSTAGE; ++s) {
            mbar_init(&bars->full[s], 1);
            mbar_init(&bars->empty[s], 1);
        }
        mbar_init(&bars->cfull, 1);
        for (int b = 0; b < 2; ++b) {
            mbar_init(&bars->tfull[b], 1);
            mbar_init(&bars->tempty[b], 4);
        }
        bars->abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __shared__ uint32_t s_hmax;
    if (threadIdx.x == 0) s_hmax = 0u;
    __syncthreads();
    after_previous_kernel();
    next_kernel_may_start();
    for (int t = threadIdx.x; t < BN; t += blockDim.x) {
        const float hn = P.hn[t]; // +inf beyond k
        if (t < P.k) atomicMax(&s_hmax, __float_as_uint(fmaxf(hn, 0.0f))); // the largest half norm (NaN counts as 0)
        hn_s[t] = hn;
        const bool pad = !(hn < VQB_DENSE_INF);
        const float hh = pad ? 1e30f : tf32_round(hn), hl = pad ? 0.0f : tf32_round(hn - hh);
        unsigned char *rowp = bh_smem + (size_t)(t >> 3) * 256 + (size_t)(t & 7) * 32;
        const int sw = ((t >> 2) & 1) * 16; // 32B swizzle: the two 16-byte halves of a row swap when bit 2 of the row is set
        *reinterpret_cast<float4 *>(rowp + sw) = make_float4(-hh, -hl, 0.0f, 0.0f);
        *reinterpret_cast<float4 *>(rowp + (16 - sw)) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (t < BM) {
            unsigned char *ap = a1_smem + (size_t)(t >> 3) * 256 + (size_t)(t & 7) * 32;
            *reinterpret_cast<float4 *>(ap + sw) = make_float4(1.0f, 1.0f, 0.0f, 0.0f);
            *reinterpret_cast<float4 *>(ap + (16 - sw)) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); // generic writes -> visible to the MMA's reads
    if (warp == 1) { // tensor memory: 512 columns = two 128 x 256 f32 accumulators
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bars->tmem_base)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem_base = bars->tmem_base;

    if (warp == 0) {
        // ------------------------------------------------ TMA producer
        if (lane == 0) {
            mbar_expect_tx(&bars->cfull, (uint32_t)kchunks * C_CHUNK_BYTES);
            for (int kc = 0; kc < kchunks; ++kc) tma_load_2d(c_smem + (size_t)kc * C_CHUNK_BYTES, &map_c, kc * CHUNK, 0, &bars->cfull);
            uint32_t it = 0;
            for (unsigned long long tile = blockIdx.x; tile < n_tiles && !*abort_flag; tile += gridDim.x) {
                for (int kc = 0; kc < kchunks; ++kc, ++it) {
                    const int s = it % NSTAGE;
                    const uint32_t use = it / NSTAGE;
                    if (!mbar_wait(&bars->empty[s], (use & 1u) ^ 1u, abort_flag, P.error, 1)) break;
                    mbar_expect_tx(&bars->full[s], X_STAGE_BYTES);
                    tma_load_2d(x_smem + (size_t)s * X_STAGE_BYTES, &map_x, kc * CHUNK, (int)(tile * BM), &bars->full[s]);
                }
            }
            if (*abort_flag) {
                // gave up: let the copies already in flight land before the CTA retires (bounded; a phase the MMA warp
                // already consumed simply runs this short wait out)
                for (uint32_t back = 0; back < NSTAGE && back < it; ++back) {
                    const uint32_t j = it - 1 - back;
                    const uint32_t addr = smem_u32(&bars->full[j % NSTAGE]);
                    for (uint32_t spin = 0; spin < 20000u; ++spin) {
                        uint32_t done;
                        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}"
                                     : "=r"(done)
                                     : "r"(addr), "r"((j / NSTAGE) & 1u)
                                     : "memory");
                        if (done) break;
                    }
                }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        if (lane == 0) {
            bool ok = mbar_wait(&bars->cfull, 0, abort_flag, P.error, 2);
            const uint64_t adesc0 = smem_desc_sw128(smem_u32(x_smem)), bdesc0 = smem_desc_sw128(smem_u32(c_smem));
            auto book_step = [](int step) { return (uint64_t)((step >> 2) * (int)(C_CHUNK_BYTES >> 4) + 2 * (step & 3)); }; // K step of the codebook's image
            uint32_t it = 0, local = 0;
            for (unsigned long long tile = blockIdx.x; ok && tile < n_tiles && !*abort_flag; tile += gridDim.x, ++local) {
                const uint32_t b = local & 1u, buse = local >> 1;
                if (!mbar_wait(&bars->tempty[b], (buse & 1u) ^ 1u, abort_flag, P.error, 3)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d_tmem = tmem_base + b * BN;
#pragma unroll
                for (int kc = 0; kc < kchunks; ++kc, ++it) {
                    const int s = it % NSTAGE;
                    const uint32_t use = it / NSTAGE;
                    if (!mbar_wait(&bars->full[s], use & 1u, abort_flag, P.error, 4)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t adesc = adesc0 + (uint64_t)(s * (int)(X_STAGE_BYTES >> 4));
#pragma unroll
                    for (int i = 0; i < 4; ++i) { // 16 values = 32 bytes = 2 descriptor units per step
                        const int j = 4 * kc + i;
                        if (j < KS) { // h.ch and h.cl
                            umma_f16(d_tmem, adesc + 2 * i, bdesc0 + book_step(j), j ? 1u : 0u);
                            umma_f16(d_tmem, adesc + 2 * i, bdesc0 + book_step(KS + j), 1u);
                        } else if (j < 2 * KS) { // l.ch
                            umma_f16(d_tmem, adesc + 2 * i, bdesc0 + book_step(j - KS), 1u);
                        }
                    }
                    umma_commit(&bars->empty[s]); // the stage is free once these MMAs have read it
                }
                if (ok) {
                    umma_tf32(d_tmem, smem_desc_sw32(smem_u32(a1_smem)), smem_desc_sw32(smem_u32(bh_smem)), 1u); // D = x.c - hn
                    umma_commit(&bars->tfull[b]);
                }
            }
        }
    } else {
        // ------------------------------------------------ epilogue: one row per lane
        const int q = warp & 3; // TMEM lane quadrant this warp may read
        const float cmax = sqrtf(2.0f * __uint_as_float(s_hmax)) * 1.00002f;
        // in the frame: what underflows in the reference's products, and distances that could overflow there
        const float s2 = P.frame[FRAME_SCALE] * P.frame[FRAME_SCALE], tiny = 1e-36f * s2, huge = fminf(1e37f * s2, 1e37f);
        unsigned long long cand_total = 0, full_scans = 0, rows_done = 0;
        bool moved = false;
        uint32_t local = 0;
        for (unsigned long long tile = blockIdx.x; tile < n_tiles && !*abort_flag; tile += gridDim.x, ++local) {
            const uint32_t b = local & 1u, buse = local >> 1;
            if (!mbar_wait(&bars->tfull[b], buse & 1u, abort_flag, P.error, 5)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const unsigned long long row = tile * BM + 32ull * q + lane;
            const bool valid = row < P.n;
            const uint32_t taddr = tmem_base + ((uint32_t)(32 * q) << 16) + b * BN;
            const float xn2 = valid ? P.xnorm2[row] : 0.0f;
            const int old_code = (P.codes && valid) ? (int)P.codes[row] : 0; // asked for now, needed after the two passes

            // pass 1: the largest D = v.c - hn, i.e. the smallest score S = -D, as the maxima of the 16 blocks of 16 consecutive columns and
            // of the 16 classes of columns equal modulo 16 (one 3-input maximum per score; columns beyond k hold -1e30)
            float hb[16], ga[16];
            bool col0_nan = false;
#pragma unroll
            for (int c = 0; c < BN / 32; ++c) {
                uint32_t ra[32];
                tmem_ld32_issue(taddr + c * 32, ra);
                tmem_wait();
                if (c == 0) col0_nan = !(__uint_as_float(ra[0]) == __uint_as_float(ra[0]));
                if (P.debug_dots && valid) {
#pragma unroll
                    for (int t = 0; t < 32; ++t) P.debug_dots[row * BN + c * 32 + t] = (c * 32 + t < P.k) ? (__uint_as_float(ra[t]) + hn_s[c * 32 + t]) / s2 : 0.0f;
                }
#pragma unroll
                for (int t = 0; t < 16; ++t)
                    ga[t] = c ? max3f(ga[t], __uint_as_float(ra[t]), __uint_as_float(ra[16 + t])) : fmaxf(__uint_as_float(ra[t]), __uint_as_float(ra[16 + t]));
                float b0 = __uint_as_float(ra[0]), b1 = __uint_as_float(ra[16]);
#pragma unroll
                for (int t = 1; t < 15; t += 2) {
                    b0 = max3f(b0, __uint_as_float(ra[t]), __uint_as_float(ra[t + 1]));
                    b1 = max3f(b1, __uint_as_float(ra[16 + t]), __uint_as_float(ra[16 + t + 1]));
                }
                hb[2 * c] = fmaxf(b0, __uint_as_float(ra[15]));
                hb[2 * c + 1] = fmaxf(b1, __uint_as_float(ra[31]));
            }
            float top = hb[0];
#pragma unroll
            for (int i = 1; i < 15; i += 2) top = max3f(top, hb[i], hb[i + 1]);
            const float best = -fmaxf(top, hb[15]); // smallest score
            // E as above with max_j |c_j| (+ the rounding of the half norms: 10 operations in a tree, split into two TF32 numbers);
            // limit = best + 2E + 1.05 (dim + 6) u (|x|^2 + 2 best + 2E) + rounding slack of the comparison itself
            const float xn = sqrtf(xn2), e2 = 2.0f * (7e-6f * xn * cmax + 4e-7f * (xn + cmax)) + 1.2e-6f * cmax * cmax;
            const float d_a = fmaxf(xn2 + 2.0f * best + e2, 0.0f);
            const float limit = best + e2 + 1.05f * (float)(P.dim + 6) * 5.9604645e-8f * d_a + 2.4e-7f * (fabsf(best) + e2) + tiny;
            const float lim_d = -limit; // centroid j is a candidate when D_j >= lim_d
            // a row the comparisons cannot rank (NaN / infinity somewhere, or centroid 0 not comparable, on which the
            // reference's scan depends) is handed over with every centroid marked
            // (also when a true distance could overflow f32: then the reference's own comparisons see infinities)
            const bool scan_all = col0_nan || !(best == best) || !(limit == limit) || !(fabsf(limit) < VQB_DENSE_INF) || !(xn2 + cmax * cmax < huge);


            // Exactly one block maximum and one class maximum at or above lim_d <=> exactly one score is (two would differ in their block
            // or in their class).  t = sat((D - lim) 2^p) is exactly 0 or 1 with lim one unit below lim_d and p such that lim 2^p ~ 2^60;
            // sum t (1 + i / 512) has count and index in one number.
            const float lim = lim_d - fabsf(lim_d) * 1.1920929e-7f;
            const uint32_t eb = (__float_as_uint(lim) >> 23) & 0xFFu;
            const float big = __uint_as_float((314u - eb) << 23), lb = -lim * big; // 2^(60 - exponent(lim)): exact
            float tb0 = 0.0f, tb1 = 0.0f, ta0 = 0.0f, ta1 = 0.0f;
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
                tb0 = fmaf(fma_sat(hb[i], big, lb), 1.0f + (float)i * 0.001953125f, tb0);
                ta0 = fmaf(fma_sat(ga[i], big, lb), 1.0f + (float)i * 0.001953125f, ta0);
                tb1 = fmaf(fma_sat(hb[i + 1], big, lb), 1.0f + (float)(i + 1) * 0.001953125f, tb1);
                ta1 = fmaf(fma_sat(ga[i + 1], big, lb), 1.0f + (float)(i + 1) * 0.001953125f, ta1);
            }
            const float tb = tb0 + tb1, ta = ta0 + ta1;
            const int only = (int)((__float_as_uint(tb + 16383.0f) & 15u) * 16 + (__float_as_uint(ta + 16383.0f) & 15u)); // 1 + i / 512 + 16383: i in the low bits
            const bool single = P.codes && !scan_all && eb - 67u < 188u && tb >= 1.0f && ta >= 1.0f && fmaxf(tb, ta) < 1.07f && only < P.k;
            if (single && valid) {
                ++cand_total, ++rows_done;
                if (only != old_code) {
                    moved = true;
                    P.codes[row] = (uint8_t)only; // the only candidate is the reference's choice
                }
            }
            const bool open = valid && !single;
            if (!__any_sync(0xffffffffu, open)) {
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&bars->tempty[b]); // this accumulator may be overwritten
                continue;
            }

            // pass 2, for the warps with an undecided row: one bit per centroid, set when D_j >= lim_d.  The sign of (D_j - lim_d) is shifted into the word,
            // so the bits arrive in reverse order and inverted.
            uint32_t words[BN / 32], ra[32], rb[32];
            tmem_ld32_issue(taddr, ra);
            tmem_wait();
#pragma unroll
            for (int cb = 0; cb < BN / 32; cb += 2) {
                tmem_ld32_issue(taddr + (cb + 1) * 32, rb);
                uint32_t m = 0;
#pragma unroll
                for (int t = 0; t < 32; ++t) m = __funnelshift_l(__float_as_uint(__uint_as_float(ra[t]) - lim_d), m, 1);
                words[cb] = ~__brev(m);
                tmem_wait();
                if (cb + 2 < BN / 32) tmem_ld32_issue(taddr + (cb + 2) * 32, ra);
                m = 0;
#pragma unroll
                for (int t = 0; t < 32; ++t) m = __funnelshift_l(__float_as_uint(__uint_as_float(rb[t]) - lim_d), m, 1);
                words[cb + 1] = ~__brev(m);
                tmem_wait();
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->tempty[b]); // this accumulator may be overwritten
            bool listed = false;
            if (open) {
                int cnt = 0;
#pragma unroll
                for (int wd = 0; wd < BN / 32; ++wd) {
                    const int lo = wd * 32;
                    const uint32_t in_range = (P.k >= lo + 32) ? 0xFFFFFFFFu : ((P.k > lo) ? ((1u << (P.k - lo)) - 1u) : 0u);
                    words[wd] = scan_all ? in_range : (words[wd] & in_range);
                    cnt += __popc(words[wd]);
                }
                if (scan_all) ++full_scans;
                else cand_total += cnt;
                ++rows_done;
                if (P.codes && cnt == 1) {
                    // the only candidate is the reference's choice (an unrankable row comes with all k >= 2 bits set)
                    int best_j = 0;
#pragma unroll
                    for (int wd = 0; wd < BN / 32; ++wd)
                        if (words[wd]) best_j = wd * 32 + __ffs(words[wd]) - 1;
                    if (best_j != old_code) {
                        moved = true;
                        P.codes[row] = (uint8_t)best_j;
                    }
                } else {
                    uint4 *o = reinterpret_cast<uint4 *>(P.cand + row * 8);
                    o[0] = make_uint4(words[0], words[1], words[2], words[3]);
                    o[1] = make_uint4(words[4], words[5], words[6], words[7]);
                    listed = P.codes != nullptr;
                }
            }
            if (P.codes) { // the rows that need the exact decision, appended in one step per warp
                const unsigned bal = __ballot_sync(0xffffffffu, listed);
                if (bal) {
                    uint32_t base = 0;
                    if (lane == 0) base = atomicAdd(P.list_count, (uint32_t)__popc(bal));
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (listed) P.list[base + __popc(bal & ((1u << lane) - 1u))] = (uint32_t)row;
                }
            }
        }
        if (P.codes && P.changed && __any_sync(0xffffffffu, moved) && lane == 0) atomicOr(P.changed, VQB_MOVED_BITS);
        if (P.stats) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                cand_total += __shfl_xor_sync(0xffffffffu, cand_total, o);
                full_scans += __shfl_xor_sync(0xffffffffu, full_scans, o);
                rows_done += __shfl_xor_sync(0xffffffffu, rows_done, o);
            }
            if (lane == 0) {
                atomicAdd(P.stats + 0, rows_done);
                atomicAdd(P.stats + 1, cand_total);
                atomicAdd(P.stats + 2, full_scans);
            }
        }
    }

    // ---------------------------------------------------- teardown
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

// The frame from a sample of 256 rows (or residuals x - centroid): eight groups of 32 rows, the median of the groups' means per
// dimension and the median of the groups' largest norms, so that a few wild rows do not move it.  Only precision depends on
// it.  s maps that norm to [32, 64): binary16 then reaches a thousand times further up, and its l parts stay normal.
__device__ __forceinline__ float upper_median8(float (&v)[8])
{
#pragma unroll
    for (int i = 1; i < 8; ++i)
#pragma unroll
        for (int j = 7; j >= i; --j) {
            const float lo = fminf(v[j - 1], v[j]), hi = fmaxf(v[j - 1], v[j]);
            v[j - 1] = lo, v[j] = hi;
        }
    return v[4];
}

__global__ void __launch_bounds__(1024) dense_frame_kernel(const float *__restrict__ x, unsigned long long n, int dim, const float *__restrict__ book,
                                                           const uint8_t *__restrict__ codes, int center, float *frame)
{
    __shared__ float s_mean[8][128], s_sq[8][32][4], s_big[8], s_mu[128];
    const int d = threadIdx.x & 127, g = threadIdx.x >> 7, lane = threadIdx.x & 31, quarter = d >> 5;
    float v[32], sum = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        const unsigned long long row = (unsigned long long)(g * 32 + i) * n / 256;
        float t = d < dim ? x[row * dim + d] : 0.0f;
        if (codes && d < dim) t -= book[(size_t)codes[row] * dim + d];
        v[i] = fabsf(t) < VQB_DENSE_INF ? t : 0.0f; // what is not finite has no say
        sum += v[i] * 0.03125f;
    }
    s_mean[g][d] = sum;
    __syncthreads();
    if (g == 0) {
        float m[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) m[i] = s_mean[i][d];
        const float mu = center ? upper_median8(m) : 0.0f;
        s_mu[d] = fabsf(mu) < VQB_DENSE_INF ? mu : 0.0f;
        frame[d] = s_mu[d];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        float a = d < dim ? v[i] - s_mu[d] : 0.0f;
        a *= a;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0) s_sq[g][i][quarter] = a;
    }
    __syncthreads();
    if (d < 32) {
        const float a = s_sq[g][d][0] + s_sq[g][d][1] + s_sq[g][d][2] + s_sq[g][d][3];
        const uint32_t big = __reduce_max_sync(0xffffffffu, a < VQB_DENSE_INF ? __float_as_uint(a) : 0u);
        if (d == 0) s_big[g] = __uint_as_float(big);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float m[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) m[i] = s_big[i];
        const float norm = sqrtf(upper_median8(m));
        const int e = norm > 0.0f && norm < VQB_DENSE_INF ? 5 - ilogbf(norm) : 0;
        frame[FRAME_SCALE] = ldexpf(1.0f, max(-40, min(40, e)));
    }
}

// A warp per centroid: image and half norm (zeros and +inf at and beyond k)
__global__ void __launch_bounds__(256) dense_codebook_kernel(const float *c, int k, int dim, int dimp, const float *frame, uint16_t *image, float *hn)
{
    after_previous_kernel();
    next_kernel_may_start();
    const int j = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const bool in = j < k;
    float v[4]; // (ordinary loads: a centroid update may come directly before)
#pragma unroll
    for (int e = 0; e < 4; ++e) v[e] = in && 4 * lane + e < dim ? c[(size_t)j * dim + 4 * lane + e] : 0.0f;
    store_codebook_row(image, hn, dimp, j, v, load_frame(frame, lane), in, lane);
}

// Images and (upper bounds of the) squared norms of the rows: one read, one write of the same size.  L lanes per row (8, 16 or
// 32), four values each, so that a warp's loads and stores are whole lines.
template <int L, bool VEC>
__global__ void __launch_bounds__(256) dense_prepare_kernel(const float *__restrict__ x, unsigned long long n, int dim, int dimp, const float *frame,
                                                            uint16_t *image, float *norms)
{
    const int lane = threadIdx.x & 31, piece = lane % L;
    const FramePiece f = load_frame(frame, piece);
    const unsigned long long step = (unsigned long long)gridDim.x * (256 / L);
    for (unsigned long long row = blockIdx.x * (unsigned long long)(256 / L) + threadIdx.x / L; row - threadIdx.x / L < n; row += step) {
        float v[4];
        load_piece<VEC>(v, x, row, piece, row < n, dim);
        float a = store_image(image + (size_t)row * 2 * dimp, dimp, piece, v, f, row < n);
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (row < n && piece == 0) norms[row] = a * 1.00001f; // an upper bound is what the shortlist needs
    }
}

CUtensorMap make_map(const uint16_t *image, unsigned long long rows, int dimp, int box_rows)
{
    return make_tensor_map_2d(image, 2 * (unsigned long long)dimp, rows, CHUNK, (unsigned)box_rows, CU_TENSOR_MAP_SWIZZLE_128B);
}

} // namespace

bool dense_tc_applicable(size_t dim, size_t k, int metric)
{
    return (metric == M_SQ || metric == M_EUCLID) && dim > 16 && dim <= 128 && k >= 2 && k <= 256;
}

size_t dense_tc_smem_bytes()
{
    return 1024 + (size_t)MAX_KCHUNKS * C_CHUNK_BYTES + (size_t)NSTAGE * X_STAGE_BYTES + BN * sizeof(float) + (size_t)(BM + BN) * 32 + sizeof(Barriers) + 64;
}

void dense_frame(CudaDevice &dev, const DenseWork &w, const float *x, size_t n, size_t dim, const float *codebook, const uint8_t *codes, bool center)
{
    if (n == 0) return;
    KernelScope ks(dev, "dense_frame");
    dense_frame_kernel<<<1, 1024, 0, dev.stream()>>>(x, n, (int)dim, codebook, codes, center ? 1 : 0, w.frame);
    VQB_CUDA_CHECK(cudaGetLastError());
    dev.count_launch();
}

void dense_prepare(CudaDevice &dev, const DenseWork &w, const float *x, size_t n, size_t dim)
{
    if (n == 0) return;
    KernelScope ks(dev, "dense_prepare");
    const int dimp = (int)dense_padded(dim);
    const bool vec = dim % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
    auto go = [&](auto kernel, int lanes) {
        const unsigned grid = (unsigned)std::max<size_t>(1, std::min<size_t>((n * lanes + 255) / 256, (size_t)dev.sm_count() * 32));
        kernel<<<grid, 256, 0, dev.stream()>>>(x, n, (int)dim, dimp, w.frame, w.image, w.norms);
    };
    if (dimp <= 32) vec ? go(dense_prepare_kernel<8, true>, 8) : go(dense_prepare_kernel<8, false>, 8);
    else if (dimp <= 64) vec ? go(dense_prepare_kernel<16, true>, 16) : go(dense_prepare_kernel<16, false>, 16);
    else vec ? go(dense_prepare_kernel<32, true>, 32) : go(dense_prepare_kernel<32, false>, 32);
    VQB_CUDA_CHECK(cudaGetLastError());
    dev.count_launch();
}

void dense_shortlist(CudaDevice &dev, const DenseWork &w, size_t n, size_t dim, const float *codebook, size_t k, unsigned long long *stats,
                     int *error_word, float *debug_dots, const ShortlistTrain *train, bool book_there)
{
    if (n == 0) return;
    const int dimp = (int)dense_padded(dim);
    if (!book_there) {
        KernelScope ks(dev, "dense_codebook");
        launch_following(dense_codebook_kernel, BN / 8, 256, 0, dev.stream(), codebook, (int)k, (int)dim, dimp, w.frame, w.book_image, w.half_norms);
        dev.count_launch();
    }
    const CUtensorMap mx = make_map(w.image, n, dimp, BM);
    const CUtensorMap mc = make_map(w.book_image, BN, dimp, BN);
    ShortlistParams p;
    p.n = n;
    p.dim = (int)dim;
    p.k = (int)k;
    p.hn = w.half_norms;
    p.frame = w.frame;
    p.xnorm2 = w.norms;
    p.cand = w.cand;
    p.stats = stats;
    p.debug_dots = debug_dots;
    p.error = error_word;
    p.codes = train ? train->codes : nullptr;
    p.changed = train ? train->changed : nullptr;
    p.list = w.list;
    p.list_count = w.list_count;
    const size_t smem = dense_tc_smem_bytes();
    const unsigned long long tiles = (n + BM - 1) / BM;
    const unsigned grid = (unsigned)std::min<unsigned long long>(tiles, (unsigned long long)dev.sm_count());
    KernelScope ks(dev, "dense_shortlist");
    auto go = [&](auto kernel) {
        VQB_CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        launch_following(kernel, grid, 192, smem, dev.stream(), mx, mc, p);
    };
    switch (dimp / 16) {
    case 2: go(dense_shortlist_kernel<2>); break;
    case 3: go(dense_shortlist_kernel<3>); break;
    case 4: go(dense_shortlist_kernel<4>); break;
    case 5: go(dense_shortlist_kernel<5>); break;
    case 6: go(dense_shortlist_kernel<6>); break;
    case 7: go(dense_shortlist_kernel<7>); break;
    default: go(dense_shortlist_kernel<8>); break;
    }
    dev.count_launch();
}

} // namespace vqb
