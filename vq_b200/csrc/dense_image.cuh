// dense_image.cuh -- rows as the tensor-core shortlist reads them (dense_tc.cu): v = s (x - mu) in two binary16 numbers, all h
// parts first, then all l parts, both padded with zeros to `dimp` values.  mu and s ("frame", 129 floats) are the same for
// rows and centroids, so distances only scale.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace vqb {

constexpr int FRAME_SCALE = 128; // frame[0 .. 127]: mu, frame[128]: s, a power of two

// values 4 * piece .. 4 * piece + 3 of a row (zeros where there are none)
template <bool VEC> __device__ __forceinline__ void load_piece(float (&v)[4], const float *x, unsigned long long row, int piece, bool in, int dim)
{
    if (VEC) {
        const float4 t = in && 4 * piece < dim ? __ldg(reinterpret_cast<const float4 *>(x + row * dim) + piece) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = in && 4 * piece + e < dim ? __ldg(x + row * dim + 4 * piece + e) : 0.0f;
    }
}

struct FramePiece {
    float mu[4], s;
};

// the frame for a lane's four dimensions (mu is zero beyond dim)
__device__ __forceinline__ FramePiece load_frame(const float *frame, int piece)
{
    FramePiece f;
    const float4 t = *reinterpret_cast<const float4 *>(frame + 4 * piece);
    f.mu[0] = t.x, f.mu[1] = t.y, f.mu[2] = t.z, f.mu[3] = t.w;
    f.s = frame[FRAME_SCALE];
    return f;
}

// Writes a lane's part of a row's image and returns its share of |v|^2.  A value beyond binary16's range becomes infinite (its l
// part NaN), which sends the row to the full scan.
__device__ __forceinline__ float store_image(uint16_t *row_image, int dimp, int piece, const float (&x)[4], const FramePiece &f, bool in)
{
    uint32_t h[2], l[2];
    float a = 0.0f;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const float v0 = (x[2 * e] - f.mu[2 * e]) * f.s, v1 = (x[2 * e + 1] - f.mu[2 * e + 1]) * f.s;
        a = fmaf(v0, v0, fmaf(v1, v1, a));
        const __half h0 = __float2half_rn(v0), h1 = __float2half_rn(v1);
        const __half l0 = __float2half_rn(v0 - __half2float(h0)), l1 = __float2half_rn(v1 - __half2float(h1));
        h[e] = (uint32_t)__half_as_ushort(h0) | ((uint32_t)__half_as_ushort(h1) << 16);
        l[e] = (uint32_t)__half_as_ushort(l0) | ((uint32_t)__half_as_ushort(l1) << 16);
    }
    if (in && 4 * piece < dimp) {
        *reinterpret_cast<uint2 *>(row_image + 4 * piece) = make_uint2(h[0], h[1]);
        *reinterpret_cast<uint2 *>(row_image + dimp + 4 * piece) = make_uint2(l[0], l[1]);
    }
    return a;
}

// What an assignment pass needs of the centroids, for a kernel that has them at hand.
struct DenseOperand {
    const float *frame;
    uint16_t *image; // null: nothing to write
    float *half_norms;
    int dimp;
};

// A warp writes image and half norm of centroid j (zeros and +inf where there is none)
__device__ __forceinline__ void store_codebook_row(uint16_t *image, float *half_norms, int dimp, int j, const float (&v)[4], FramePiece f, bool in, int lane)
{
    if (!in) f.mu[0] = f.mu[1] = f.mu[2] = f.mu[3] = 0.0f;
    float a = store_image(image + (size_t)j * 2 * dimp, dimp, lane, v, f, true);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) half_norms[j] = in ? 0.5f * a : __int_as_float(0x7f800000);
}

} // namespace vqb
