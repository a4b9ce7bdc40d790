// resolve.cu -- exact decision among shortlisted centroids (the second half of the tensor-core path, dense_tc.cu) and what the
// residual quantizer does once a row's centroid is known (src/rvq.rs:111-138, 186-213).
#include <algorithm>
#include <type_traits>

#include "cuda_device.hpp"
#include "dense_image.cuh"
#include "dense_tc.hpp"
#include "kernels_common.cuh"

namespace vqb {

namespace {

// One warp per listed row, one lane per candidate: each candidate's distance in the reference's own f32 arithmetic
// (src/vector.rs:198-220, src/distances.rs:130-140), the smallest with the lowest index wins.  The shortlist leaves few rows (a
// hundredth of a Gaussian mixture's; more only where centroids coincide, and then a warp's lanes are full), so the time is
// the way to a few centroids in L2: 16 loads per lane are on their way at once.
template <bool VEC>
__global__ void __launch_bounds__(256) resolve_kernel(const float *__restrict__ x, int dim, int k, const float *__restrict__ book, int euclid,
                                                      const uint32_t *cand, const uint32_t *list, uint32_t *list_count,
                                                      uint8_t *codes, uint32_t *changed)
{
    __shared__ uint8_t s_number[8][256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    after_previous_kernel();
    next_kernel_may_start();
    const uint32_t total = *list_count;
    bool moved = false;
    for (uint32_t at = blockIdx.x * 8 + warp; at < total; at += gridDim.x * 8) {
        const size_t row = list[at];
        int cnt = 0;
#pragma unroll
        for (int w = 0; w < DENSE_MASK_WORDS; ++w) {
            const uint32_t word = cand[row * DENSE_MASK_WORDS + w];
            if (word >> lane & 1u) s_number[warp][cnt + __popc(word & ((1u << lane) - 1u))] = (uint8_t)(w * 32 + lane);
            cnt += __popc(word);
        }
        __syncwarp();
        const float *xr = x + row * dim;
        float best = VQB_DENSE_INF;
        int code = 0; // stays where nothing is below +inf
        bool stuck = false;
        for (int base = 0; base < cnt; base += 32) {
            const bool in = base + lane < cnt;
            const int j = s_number[warp][in ? base + lane : 0];
            const float *c = book + (size_t)j * dim;
            float d = 0.0f;
            auto add = [&](float xv, float cv) {
                const float e = __fsub_rn(xv, cv);
                d = __fadd_rn(d, __fmul_rn(e, e));
            };
            if (VEC) {
#pragma unroll 16
                for (int i = 0; i < dim; i += 4) {
                    const float4 cv = __ldg(reinterpret_cast<const float4 *>(c + i)), xv = __ldg(reinterpret_cast<const float4 *>(xr + i));
                    add(xv.x, cv.x), add(xv.y, cv.y), add(xv.z, cv.z), add(xv.w, cv.w);
                }
            } else {
#pragma unroll 16
                for (int i = 0; i < dim; ++i) add(__ldg(xr + i), __ldg(c + i));
            }
            if (euclid) d = __fsqrt_rn(d);
            stuck = stuck || __any_sync(0xffffffffu, in && j == 0 && !(d == d)); // the reference's scan starts at centroid 0: a NaN there stays
            float low = in && d < VQB_DENSE_INF ? d : VQB_DENSE_INF;
            const float mine = low;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) low = fminf(low, __shfl_xor_sync(0xffffffffu, low, o));
            const int jm = (int)__reduce_min_sync(0xffffffffu, mine == low ? (unsigned)j : 0xFFFFFFFFu);
            if (low < best) best = low, code = jm; // candidates ascend: an equal distance later on loses
        }
        if (stuck) code = 0;
        if (lane == 0 && codes[row] != (uint8_t)code) {
            moved = true;
            codes[row] = (uint8_t)code;
        }
        __syncwarp();
    }
    if (lane == 0 && moved && changed) atomicOr(changed, VQB_MOVED_BITS);
    // the list is empty again for the next pass (a memset between two passes of few rows took 4 us, and the overlap of their launches)
    __syncthreads();
    if (threadIdx.x == 0 && atomicAdd(list_count + 1, 1u) == gridDim.x - 1) list_count[0] = list_count[1] = 0u, list_count[2] = total;
}

// L lanes per row, four values each (as dense_prepare_kernel): one read of the rows, one write of the residuals, one of their
// images; the codebook's rows come from L2.
template <int L, bool VEC>
__global__ void __launch_bounds__(256) rvq_apply_kernel(const float *x, float *res, unsigned long long n, int dim, int dimp, const float *__restrict__ book,
                                                        const uint8_t *__restrict__ codes, double *norm_sum,
                                                        const float *frame, uint16_t *image, float *norms)
{
    const int lane = threadIdx.x & 31, piece = lane % L;
    const FramePiece f = load_frame(frame, piece);
    const unsigned long long step = (unsigned long long)gridDim.x * (256 / L);
    double total = 0.0;
    for (unsigned long long row = blockIdx.x * (unsigned long long)(256 / L) + threadIdx.x / L; row - threadIdx.x / L < n; row += step) {
        const bool in = row < n;
        float v[4], c[4];
        const int code = in ? (int)codes[row] : 0;
        if (VEC) {
            const float4 t = in && 4 * piece < dim ? *reinterpret_cast<const float4 *>(x + row * dim + 4 * piece) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = in && 4 * piece + e < dim ? x[row * dim + 4 * piece + e] : 0.0f;
        }
        load_piece<VEC>(c, book, (unsigned long long)code, piece, in, dim);
        float a = 0.0f;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            v[e] = __fsub_rn(v[e], c[e]);
            a = fmaf(v[e], v[e], a);
        }
        if (in) {
            if (VEC) {
                if (4 * piece < dim) *reinterpret_cast<float4 *>(res + row * dim + 4 * piece) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (4 * piece + e < dim) res[row * dim + 4 * piece + e] = v[e];
            }
        }
        float fa = store_image(image + (size_t)row * 2 * dimp, dimp, piece, v, f, in);
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            fa += __shfl_xor_sync(0xffffffffu, fa, o);
        }
        if (norm_sum && in && piece == 0) total += (double)sqrtf(a);
        if (in && piece == 0) norms[row] = fa * 1.00001f; // an upper bound is what the shortlist needs
    }
    if (norm_sum) { // one atomic a CTA: one a warp, on the one address, took 45 us of 58 for 33,506 rows
        __shared__ double s_total[8];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
        if (lane == 0) s_total[threadIdx.x >> 5] = total;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 1; w < 8; ++w) total += s_total[w];
            if (total != 0.0) atomicAdd(norm_sum, total);
        }
    }
}

// lanes per row that a width takes, and the kernel for them
template <typename F> void with_lanes(size_t dimp, bool vec, F &&f)
{
    if (dimp <= 32) vec ? f(std::integral_constant<int, 8>(), std::true_type()) : f(std::integral_constant<int, 8>(), std::false_type());
    else if (dimp <= 64) vec ? f(std::integral_constant<int, 16>(), std::true_type()) : f(std::integral_constant<int, 16>(), std::false_type());
    else vec ? f(std::integral_constant<int, 32>(), std::true_type()) : f(std::integral_constant<int, 32>(), std::false_type());
}

bool aligned(const void *p, unsigned bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; }

unsigned grid_rows(CudaDevice &dev, size_t n, int lanes)
{
    return (unsigned)std::max<size_t>(1, std::min<size_t>((n * lanes + 255) / 256, (size_t)dev.sm_count() * 32));
}

} // namespace

void dense_resolve(CudaDevice &dev, const DenseWork &w, const float *x, size_t n, size_t dim, const float *codebook, size_t k, bool euclid,
                   uint8_t *codes, uint32_t *changed)
{
    if (n == 0) return;
    const bool vec = dim % 4 == 0 && aligned(x, 16) && aligned(codebook, 16);
    // the number of listed rows is only known on the device
    const unsigned grid = (unsigned)std::max<size_t>(1, std::min<size_t>((n + 7) / 8, (size_t)dev.sm_count() * 6));
    KernelScope ks(dev, "dense_resolve");
    auto kernel = vec ? resolve_kernel<true> : resolve_kernel<false>;
    launch_following(kernel, grid, 256, 0, dev.stream(), x, (int)dim, (int)k, codebook, euclid ? 1 : 0, w.cand, w.list, w.list_count, codes, changed);
    dev.count_launch();
}

void rvq_apply(CudaDevice &dev, const RvqApply &a, const DenseWork &w)
{
    if (a.n == 0) return;
    const size_t dimp = dense_padded(a.dim);
    dense_frame(dev, w, a.x, a.n, a.dim, a.codebook, a.codes, true);
    KernelScope ks(dev, "rvq_apply");
    with_lanes(dimp, a.dim % 4 == 0 && aligned(a.x, 16) && aligned(a.res, 16) && aligned(a.codebook, 16), [&](auto lanes, auto vec) {
        constexpr int L = decltype(lanes)::value;
        rvq_apply_kernel<L, decltype(vec)::value><<<grid_rows(dev, a.n, L), 256, 0, dev.stream()>>>(
            a.x, a.res, a.n, (int)a.dim, (int)dimp, a.codebook, a.codes, a.norm_sum, w.frame, w.image, w.norms);
    });
    VQB_CUDA_CHECK(cudaGetLastError());
    dev.count_launch();
}

} // namespace vqb
