// svd.cu -- the sweeps of the one-sided (Hestenes) Jacobi SVD behind OPQ's Procrustes step (src/opq.rs:180-183, where the
// reference calls nalgebra's SVD) on the device.
//
// One CTA of 1024 threads.  A sweep visits all n(n-1)/2 column pairs in the round-robin (tournament) order: n - 1 steps of n/2
// disjoint pairs, one team of 1024 / (n/2) threads per pair (n = 64 or 128).  The working matrices G = A V and V are held transposed (row p =
// column p) in global memory and read / written past the L1 cache, so a step sees what the previous step wrote after one
// __syncthreads.  The sweeps end when no pair rotated (|g_p . g_q| <= 1e-15 |g_p| |g_q| for all pairs) or after 60 sweeps;
// singular values, U and the completion of a rank-deficient U are computed by the caller from the converged G.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "cuda_device.hpp"

namespace vqb {

namespace {

template <int EPT> // elements of a row per thread = n / (threads per pair)
__global__ void __launch_bounds__(1024, 1) jacobi_sweeps_kernel(double *gt, double *vt, int n, int *sweeps_out)
{
    __shared__ int rotated_any;
    const int pairs = n / 2;
    const int team = 1024 / pairs;            // threads per pair: a power of two between 8 and 32 (and at most a warp)
    const int pr = threadIdx.x / team, tl = threadIdx.x % team;
    const unsigned lane = threadIdx.x & 31u;
    const unsigned team_mask = (team == 32) ? 0xffffffffu : (((1u << team) - 1u) << (lane & ~(unsigned)(team - 1)));
    const double eps = 1e-15;
    int sweep = 0;
    for (; sweep < 60; ++sweep) {
        if (threadIdx.x == 0) rotated_any = 0;
        __syncthreads();
        for (int step = 0; step < n - 1; ++step) {
            // round-robin pairing of 0 .. n-1: player n-1 stays, the others rotate
            int p, q;
            if (pr == 0) {
                p = n - 1;
                q = step;
            } else {
                p = (step + pr) % (n - 1);
                q = (step - pr + (n - 1)) % (n - 1);
            }
            if (p > q) {
                const int t = p;
                p = q;
                q = t;
            }
            double *gp = gt + (size_t)p * n, *gq = gt + (size_t)q * n;
            double *vp = vt + (size_t)p * n, *vq = vt + (size_t)q * n;
            // this thread's elements of the two G rows stay in registers from the dot products to the rotation
            double ga[EPT], gb[EPT];
#pragma unroll
            for (int e = 0; e < EPT; ++e) {
                const int i = tl + e * team;
                ga[e] = __ldcg(gp + i), gb[e] = __ldcg(gq + i);
            }
            double alpha = 0.0, beta = 0.0, gamma = 0.0;
#pragma unroll
            for (int e = 0; e < EPT; ++e) {
                alpha += ga[e] * ga[e];
                beta += gb[e] * gb[e];
                gamma += ga[e] * gb[e];
            }
            for (int o = team >> 1; o > 0; o >>= 1) {
                alpha += __shfl_xor_sync(team_mask, alpha, o);
                beta += __shfl_xor_sync(team_mask, beta, o);
                gamma += __shfl_xor_sync(team_mask, gamma, o);
            }
            // the rotation's parameters: f64 square roots and divisions are slow, so one thread of the team computes them
            double c = 1.0, sn = 0.0;
            int rot = 0;
            if (tl == 0 && !(fabs(gamma) <= eps * sqrt(alpha * beta) || gamma == 0.0)) {
                rot = 1;
                const double zeta = (beta - alpha) / (2.0 * gamma);
                const double t = (zeta >= 0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
                c = 1.0 / sqrt(1.0 + t * t);
                sn = c * t;
            }
            const int src = (int)(lane & ~(unsigned)(team - 1));
            rot = __shfl_sync(team_mask, rot, src);
            c = __shfl_sync(team_mask, c, src);
            sn = __shfl_sync(team_mask, sn, src);
            if (rot) {
                if (tl == 0) rotated_any = 1;
#pragma unroll
                for (int e = 0; e < EPT; ++e) {
                    const int i = tl + e * team;
                    const double va = __ldcg(vp + i), vb = __ldcg(vq + i);
                    __stcg(gp + i, c * ga[e] - sn * gb[e]);
                    __stcg(gq + i, sn * ga[e] + c * gb[e]);
                    __stcg(vp + i, c * va - sn * vb);
                    __stcg(vq + i, sn * va + c * vb);
                }
            }
            __syncthreads(); // the rows written in this step are read by other teams in the next
        }
        if (!rotated_any) break;
        __syncthreads();
    }
    if (threadIdx.x == 0) *sweeps_out = sweep;
}

} // namespace

bool CudaDevice::svd_sweeps(double *gt, double *vt, size_t n)
{
    // n = 64 or 128: n/2 pairs, teams of 32 or 16 threads inside one warp, 2 or 8 elements of each row per thread
    if (n != 64 && n != 128) return false;
    const size_t bytes = sizeof(double) * n * n;
    double *g_d = static_cast<double *>(alloc(bytes)), *v_d = static_cast<double *>(alloc(bytes));
    int *sw_d = static_cast<int *>(alloc(sizeof(int)));
    upload(g_d, gt, bytes);
    upload(v_d, vt, bytes);
    {
        KernelScope ks(*this, "jacobi_sweeps");
        if (n == 64) jacobi_sweeps_kernel<2><<<1, 1024, 0, stream_>>>(g_d, v_d, (int)n, sw_d);
        else jacobi_sweeps_kernel<8><<<1, 1024, 0, stream_>>>(g_d, v_d, (int)n, sw_d);
        VQB_CUDA_CHECK(cudaGetLastError());
        count_launch();
    }
    download(gt, g_d, bytes);
    download(vt, v_d, bytes);
    release(g_d), release(v_d), release(sw_d);
    return true;
}

} // namespace vqb

// ------------------------------------------------------------------------------------------------
// The rotation without the SVD.  src/opq.rs:180-183 takes A = U S V^T and sets R = V U^T.  Since A^T = (V U^T)(U S U^T), that R
// is the orthogonal polar factor of A^T, which is unique when A has full rank and does not depend on how an SVD orders or signs
// its vectors.  The Newton-Schulz iteration
//        X_0 = A^T / sqrt(|A|_1 |A|_inf),      X_{k+1} = X_k (1.5 I - 0.5 X_k^T X_k)
// drives every singular value of X (all in (0, 1] at the start) to 1 and leaves the singular vectors alone, so it converges to
// that factor: linearly (x 1.5 per step) while a singular value is small, then quadratically.  All of it is 128 x 128 x 128 f64
// products on the device: no download of A, no sweeps on one SM.
//
// polar_iterate_kernel runs the whole iteration in ONE cooperative launch (one CTA per 16 x 16 tile, all resident; its own
// bounded barrier between the two products of a step; the residual max|X^T X - I| is looked at on the device after every
// step).  While the singular values are spread it uses, instead of (1.5, 0.5), the odd cubic a x - b x^3 that maps the current
// interval [l, 1] of singular values into the narrowest interval [l', 1] (l' is known in closed form, so every CTA follows the
// same sequence); small singular values then grow by up to 2.6 instead of 1.5 per step.  The interval starts at l = 1e-4, a
// guess: a smaller true value only means the last steps run with the plain coefficients.  One launch and about 16 steps
// replace some 25 steps of three stream operations each and a host round trip every eighth step (1.23 -> 0.37 ms at n = 128).
// A step is a chain of trips to L2 and of barriers, so a product waits for one trip (all operands of a tile requested at once; one per
// 16 values of the contraction before), the residual arrives with the next product's operands, a thread keeps its own entry of the
// iterate, the coefficients come with the launch and the barrier is a release and an acquire instead of two full fences: 0.325 -> 0.148 ms
// at n = 128 (the products alone 0.185).
// The step-by-step kernels below remain for matrices whose tiles cannot all be resident.  If the iteration has not converged
// after 96 steps (rank-deficient or extremely ill-conditioned A) the caller falls back to the Jacobi SVD, which also
// completes a null space.
// ------------------------------------------------------------------------------------------------
namespace vqb {

namespace {

constexpr int POLAR_TILE = 16;
constexpr double POLAR_TOL = 1e-13;

// scale^2 = |a|_1 |a|_inf (largest column sum times largest row sum of |a|), an upper bound of the largest singular value squared
// that is within a small factor of it
__global__ void polar_scale_kernel(const double *a, int n, double *scale2)
{
    __shared__ double red[256];
    double best_row = 0.0, best_col = 0.0;
    for (int t = threadIdx.x; t < n; t += 256) {
        double r = 0.0, c = 0.0;
        for (int u = 0; u < n; ++u) {
            r += fabs(a[(size_t)t * n + u]);
            c += fabs(a[(size_t)u * n + t]);
        }
        best_row = fmax(best_row, r);
        best_col = fmax(best_col, c);
    }
    red[threadIdx.x] = best_row;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + o]);
        __syncthreads();
    }
    const double rmax = red[0];
    __syncthreads();
    red[threadIdx.x] = best_col;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + o]);
        __syncthreads();
    }
    if (threadIdx.x == 0) *scale2 = rmax * red[0];
}

// x[i][j] = a[j][i] / sqrt(scale2)
__global__ void polar_init_kernel(const double *a, int n, const double *scale2, double *x)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * n) return;
    const int i = t / n, j = t % n;
    const double f = sqrt(*scale2);
    x[t] = (f > 0.0 && f == f) ? a[(size_t)j * n + i] / f : 0.0;
}

// b = x^T x, and *resid = max |b - I| (bits of a non-negative double, so an integer max orders them)
__global__ void __launch_bounds__(POLAR_TILE *POLAR_TILE) polar_gram_kernel(const double *x, int n, double *b, unsigned long long *resid)
{
    __shared__ double xa[POLAR_TILE][POLAR_TILE + 1], xb[POLAR_TILE][POLAR_TILE + 1];
    const int tx = threadIdx.x % POLAR_TILE, ty = threadIdx.x / POLAR_TILE;
    const int i = blockIdx.y * POLAR_TILE + ty, j = blockIdx.x * POLAR_TILE + tx; // b[i][j] = sum_r x[r][i] x[r][j]
    double acc = 0.0;
    for (int r0 = 0; r0 < n; r0 += POLAR_TILE) {
        xa[ty][tx] = x[(size_t)(r0 + ty) * n + blockIdx.y * POLAR_TILE + tx]; // rows r0.., columns of the i block
        xb[ty][tx] = x[(size_t)(r0 + ty) * n + blockIdx.x * POLAR_TILE + tx]; // rows r0.., columns of the j block
        __syncthreads();
#pragma unroll
        for (int r = 0; r < POLAR_TILE; ++r) acc = fma(xa[r][ty], xb[r][tx], acc);
        __syncthreads();
    }
    b[(size_t)i * n + j] = acc;
    const double dev = fabs(acc - (i == j ? 1.0 : 0.0));
    atomicMax(resid, (unsigned long long)__double_as_longlong(dev == dev ? dev : 1e300));
}

// y = 1.5 x - 0.5 x b    (y = x once the residual of this step's b is below the tolerance)
__global__ void __launch_bounds__(POLAR_TILE *POLAR_TILE) polar_update_kernel(const double *x, const double *b, int n, const unsigned long long *resid, double *y)
{
    __shared__ double xs[POLAR_TILE][POLAR_TILE + 1], bs[POLAR_TILE][POLAR_TILE + 1];
    const int tx = threadIdx.x % POLAR_TILE, ty = threadIdx.x / POLAR_TILE;
    const int i = blockIdx.y * POLAR_TILE + ty, j = blockIdx.x * POLAR_TILE + tx;
    if (__longlong_as_double((long long)*resid) < POLAR_TOL) {
        y[(size_t)i * n + j] = x[(size_t)i * n + j];
        return;
    }
    double acc = 0.0;
    for (int r0 = 0; r0 < n; r0 += POLAR_TILE) {
        xs[ty][tx] = x[(size_t)i * n + r0 + tx];
        bs[ty][tx] = b[(size_t)(r0 + ty) * n + j];
        __syncthreads();
#pragma unroll
        for (int r = 0; r < POLAR_TILE; ++r) acc = fma(xs[ty][r], bs[r][tx], acc);
        __syncthreads();
    }
    y[(size_t)i * n + j] = 1.5 * x[(size_t)i * n + j] - 0.5 * acc;
}

// ---- the whole iteration in one cooperative launch ---------------------------------------------
// The coefficients of the steps: the cubic a x - b x^3 that maps [l, 1] into the narrowest [l', 1], until l has reached 1; (1.5, 0.5) beyond
struct PolarSteps {
    static constexpr int N = 24;
    double a[N], b[N];
};

PolarSteps polar_steps(double l)
{
    PolarSteps st;
    for (int i = 0; i < PolarSteps::N; ++i) {
        st.a[i] = 1.5, st.b[i] = 0.5;
        if (l < 0.999) {
            const double s = 1.0 + l + l * l, xs = std::sqrt(s / 3.0);
            const double pa = 2.0 / ((2.0 / 3.0) * xs + 1.0 - 1.0 / s), pe = (2.0 * pa / 3.0) * xs - 1.0;
            st.a[i] = pa / (1.0 + pe);
            st.b[i] = pa / s / (1.0 + pe);
            l = (1.0 - pe) / (1.0 + pe);
        }
    }
    return st;
}

struct PolarWork {
    double *x0, *x1, *b;             // n x n each
    unsigned long long *resid;       // [max_steps + 1] bits of max |X^T X - I| per step, zero on entry
    unsigned long long *scale;       // [2] bits of |A|_inf and |A|_1, zero on entry
    unsigned int *arrivals;          // grid barrier counter, zero on entry
    int *status;                     // [0] 1 = converged, 0 = not, -1 = a barrier wait ran out; [1] steps taken
};

// All threads of all CTAs call this the same number of times; `round` counts the calls from 1.  Bounded: a CTA that does not
// see the others arrive gives up, records -1 and every later call returns false at once.
__device__ __forceinline__ bool polar_grid_barrier(const PolarWork &w, unsigned int round, unsigned int ctas, int *failed_sh)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        // release and acquire on the counter itself: no fence waits for anything else
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(w.arrivals) : "memory");
        const unsigned int target = round * ctas;
        for (unsigned int i = 0;;) {
            unsigned int seen;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(w.arrivals) : "memory");
            if ((int)(seen - target) >= 0) break;
            if (++i > (1u << 26) || ((i & 63u) == 0 && *reinterpret_cast<volatile int *>(w.status) < 0)) {
                *reinterpret_cast<volatile int *>(w.status) = -1;
                *failed_sh = 1;
                break;
            }
        }
    }
    __syncthreads();
    return *failed_sh == 0;
}

// Sum over r of left(r, i) * right(r, j) for the CTA's 16 x 16 tile: thread t gets entry (t / 16, t % 16).  KC values of r at a time lie in shared
// memory, all of a thread's loads of them in flight at once (one trip to L2 instead of one per 16); four groups of 64 threads take every
// fourth r with 2 x 2 entries per thread, which are added up at the end.
//   left(r, i) = TRANSPOSED ? left[(i0 + i) n + r] : left[r n + i0 + i];   right(r, j) = right[r n + j0 + j]
constexpr int POLAR_LD = POLAR_TILE + 2; // doubles of a row in shared memory: 16-byte pieces stay whole, transposed stores spread over the banks
template <int KC> struct PolarTiles {
    double l[KC][POLAR_LD], r[KC][POLAR_LD];
};

template <int KC, bool TRANSPOSED>
__device__ __forceinline__ double polar_tile(const double *left, const double *right, int n, int i0, int j0, PolarTiles<KC> &sh)
{
    constexpr int PIECES = KC * POLAR_TILE / 2 / 256; // 16-byte pieces of either operand per thread and chunk
    const int t = threadIdx.x, g = t >> 6, ti = (t >> 3) & 7, tj = t & 7;
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
    for (int r0 = 0; r0 < n; r0 += KC) {
        const int kc = min(KC, n - r0); // a multiple of 16
        double2 lv[PIECES], rv[PIECES];
#pragma unroll
        for (int u = 0; u < PIECES; ++u) {
            const int r = (t >> 3) + 32 * u;                // row of the chunk, piece t & 7 of its 128 bytes
            const int r2 = 2 * ((t & 15) + POLAR_TILE * u); // TRANSPOSED: values r2, r2 + 1 of row t / 16
            if (r < kc) rv[u] = __ldcg(reinterpret_cast<const double2 *>(right + (size_t)(r0 + r) * n + j0) + (t & 7));
            if (TRANSPOSED) {
                if (r2 < kc) lv[u] = __ldcg(reinterpret_cast<const double2 *>(left + (size_t)(i0 + (t >> 4)) * n + r0 + r2));
            } else if (r < kc) {
                lv[u] = __ldcg(reinterpret_cast<const double2 *>(left + (size_t)(r0 + r) * n + i0) + (t & 7));
            }
        }
        if (r0) __syncthreads(); // the chunk before has been used
#pragma unroll
        for (int u = 0; u < PIECES; ++u) {
            const int r = (t >> 3) + 32 * u, r2 = 2 * ((t & 15) + POLAR_TILE * u);
            if (r < kc) *reinterpret_cast<double2 *>(&sh.r[r][2 * (t & 7)]) = rv[u];
            if (TRANSPOSED) {
                if (r2 < kc) sh.l[r2][t >> 4] = lv[u].x, sh.l[r2 + 1][t >> 4] = lv[u].y;
            } else if (r < kc) {
                *reinterpret_cast<double2 *>(&sh.l[r][2 * (t & 7)]) = lv[u];
            }
        }
        __syncthreads();
#pragma unroll 4
        for (int r = g; r < kc; r += 4) {
            const double2 a = *reinterpret_cast<const double2 *>(&sh.l[r][2 * ti]), b = *reinterpret_cast<const double2 *>(&sh.r[r][2 * tj]);
            acc[0][0] = fma(a.x, b.x, acc[0][0]), acc[0][1] = fma(a.x, b.y, acc[0][1]);
            acc[1][0] = fma(a.y, b.x, acc[1][0]), acc[1][1] = fma(a.y, b.y, acc[1][1]);
        }
    }
    __syncthreads();
    double *part = reinterpret_cast<double *>(&sh); // [4][16][16]
    static_assert(4 * POLAR_TILE * POLAR_TILE * sizeof(double) <= sizeof(PolarTiles<KC>), "the partial sums fit into the operands' place");
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) part[(g * POLAR_TILE + 2 * ti + a) * POLAR_TILE + 2 * tj + b] = acc[a][b];
    __syncthreads();
    const double sum = (part[t] + part[t + 256]) + (part[t + 512] + part[t + 768]);
    __syncthreads();
    return sum;
}

// max over the CTA of a non-negative value into *out (bits of a non-negative double are ordered like integers), by thread 0, whose
// grid barrier follows
__device__ __forceinline__ void polar_max(double v, unsigned long long *out, double *red)
{
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int q = 1; q < 8; ++q) v = fmax(v, red[q]);
        atomicMax(out, (unsigned long long)__double_as_longlong(v));
    }
}

template <int KC, int CTAS_PER_SM>
__global__ void __launch_bounds__(POLAR_TILE *POLAR_TILE, CTAS_PER_SM)
    polar_iterate_kernel(const double *a, int dim, int n, PolarWork w, float *rot, int max_steps, const __grid_constant__ PolarSteps steps)
{
    // dim: the matrix as it is; n: whole tiles.  The rows and columns beyond it are zeros, which every step leaves zeros, and do not count as
    // missing from the identity.
    __shared__ __align__(16) PolarTiles<KC> tiles;
    __shared__ double red[8];
    __shared__ int failed_sh;
    const int i0 = blockIdx.y * POLAR_TILE, j0 = blockIdx.x * POLAR_TILE;
    const int i = i0 + threadIdx.x / POLAR_TILE, j = j0 + threadIdx.x % POLAR_TILE;
    const unsigned int ctas = gridDim.x * gridDim.y;
    unsigned int round = 0;
    if (threadIdx.x == 0) failed_sh = 0;
    // scale^2 = |a|_1 |a|_inf: a warp per row sum or column sum
    double best[2] = {0.0, 0.0};
    for (unsigned int v = (blockIdx.y * gridDim.x + blockIdx.x) * 8u + (threadIdx.x >> 5); v < 2u * (unsigned)dim; v += 8u * ctas) {
        const bool column = v >= (unsigned)dim;
        const size_t first = column ? v - (unsigned)dim : (size_t)v * dim, step = column ? (size_t)dim : 1;
        double sum = 0.0;
#pragma unroll 4
        for (int u = threadIdx.x & 31; u < dim; u += 32) sum += fabs(__ldcg(a + first + u * step));
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        best[column] = fmax(best[column], sum); // (a NaN is passed over)
    }
    double *cur = w.x0, *nxt = w.x1;
    const bool inside = i < dim && j < dim;
    double own = inside ? __ldcg(a + (size_t)j * dim + i) : 0.0; // this thread's entry of the iterate; X_0 = A^T inv, the factor applied in step 0
    cur[(size_t)i * n + j] = own;
    polar_max(best[0], w.scale, red);
    __syncthreads();
    polar_max(best[1], w.scale + 1, red);
    if (!polar_grid_barrier(w, ++round, ctas, &failed_sh)) return;
    const double f = sqrt(__longlong_as_double((long long)__ldcg(w.scale)) * __longlong_as_double((long long)__ldcg(w.scale + 1)));
    double inv = (f > 0.0 && f == f) ? 1.0 / f : 0.0;
    double resid = 1.0;
    int step = 0;
    for (; step <= max_steps; ++step) {
        // b = X^T X, tile (i-block, j-block), and the step's residual
        const double b = polar_tile<KC, false>(cur, cur, n, i0, j0, tiles) * inv * inv;
        w.b[(size_t)i * n + j] = b;
        const double dev = fabs(b - (i == j && inside ? 1.0 : 0.0));
        polar_max(dev == dev ? dev : 1e300, w.resid + step, red);
        if (!polar_grid_barrier(w, ++round, ctas, &failed_sh)) return;
        // nxt = ca X - cb X b, tile (i-block, j-block); the residual arrives with its operands
        const unsigned long long bits = __ldcg(w.resid + step);
        const double xb = polar_tile<KC, true>(cur, w.b, n, i0, j0, tiles);
        resid = __longlong_as_double((long long)bits);
        if (resid < POLAR_TOL || step == max_steps) break; // the same value in every CTA
        const double ca = step < PolarSteps::N ? steps.a[step] : 1.5, cb = step < PolarSteps::N ? steps.b[step] : 0.5;
        own = (ca * own - cb * xb) * inv;
        nxt[(size_t)i * n + j] = own;
        inv = 1.0;
        if (!polar_grid_barrier(w, ++round, ctas, &failed_sh)) return;
        double *t = cur;
        cur = nxt;
        nxt = t;
    }
    if (inside) rot[(size_t)i * dim + j] = (float)(own * inv);
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        w.status[0] = resid < 1e-11 ? 1 : 0;
        w.status[1] = step;
    }
}

__global__ void polar_finish_kernel(const double *x, int count, float *rot)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < count) rot[t] = (float)x[t];
}

} // namespace

bool CudaDevice::polar_rotation(const double *a_dev, size_t dim, float *rot_dev)
{
    if (dim == 0 || dim > 512) return false;
    const size_t n = (dim + POLAR_TILE - 1) / POLAR_TILE * POLAR_TILE;
    const size_t bytes = sizeof(double) * n * n;
    const int max_steps = 96;
    {
        // one cooperative launch when every tile's CTA can be resident at once
        int per_sm = 0, coop = 0, dev_id = 0;
        cudaGetDevice(&dev_id);
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev_id);
        // 128 values of the contraction at a time while all CTAs fit beside each other with the registers that takes (n <= 272 on 148 SMs), else 32
        const size_t ctas = (n / POLAR_TILE) * (n / POLAR_TILE);
        auto kernel = polar_iterate_kernel<128, 2>;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, POLAR_TILE * POLAR_TILE, 0);
        if ((size_t)per_sm * (size_t)sm_count() < ctas) {
            kernel = polar_iterate_kernel<32, 7>;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, POLAR_TILE * POLAR_TILE, 0);
        }
        if (coop && (size_t)per_sm * (size_t)sm_count() >= ctas && std::getenv("VQB_POLAR_STEPWISE") == nullptr) {
            const size_t extra = sizeof(unsigned long long) * (max_steps + 4) + 64;
            unsigned char *blk = static_cast<unsigned char *>(alloc(3 * bytes + extra));
            PolarWork w;
            w.x0 = reinterpret_cast<double *>(blk);
            w.x1 = w.x0 + n * n;
            w.b = w.x1 + n * n;
            w.resid = reinterpret_cast<unsigned long long *>(blk + 3 * bytes);
            w.scale = w.resid + max_steps + 2;
            w.arrivals = reinterpret_cast<unsigned int *>(w.scale + 2);
            w.status = reinterpret_cast<int *>(w.arrivals + 2);
            int status[2] = {0, 0};
            {
                KernelScope ks(*this, "polar_rotation");
                VQB_CUDA_CHECK(cudaMemsetAsync(w.resid, 0, extra, stream_));
                const dim3 grid((unsigned)(n / POLAR_TILE), (unsigned)(n / POLAR_TILE));
                int dim_i = (int)dim, n_i = (int)n, steps_i = max_steps;
                PolarSteps steps = polar_steps(1e-4);
                void *args[] = {(void *)&a_dev, (void *)&dim_i, (void *)&n_i, (void *)&w, (void *)&rot_dev, (void *)&steps_i, (void *)&steps};
                VQB_CUDA_CHECK(cudaLaunchCooperativeKernel((const void *)kernel, grid, dim3(POLAR_TILE * POLAR_TILE), args, 0, stream_));
                count_launch();
            }
            download(status, w.status, sizeof status);
            release(blk);
            if (status[0] < 0) throw Error(100, "polar rotation: a wait between the steps ran out");
            return status[0] == 1;
        }
    }
    if (dim != n) return false; // the launches below take whole tiles
    double *x0 = static_cast<double *>(alloc(bytes)), *x1 = static_cast<double *>(alloc(bytes)), *b = static_cast<double *>(alloc(bytes));
    double *fro2 = static_cast<double *>(alloc(sizeof(double)));
    unsigned long long *resid = static_cast<unsigned long long *>(alloc(sizeof(unsigned long long) * 2));
    const int count = (int)(n * n);
    const dim3 grid((unsigned)(n / POLAR_TILE), (unsigned)(n / POLAR_TILE));
    const int batch = 8; // x 1.5 per step while a singular value is small: down to 1e-16 of the largest
    double *cur = x0, *nxt = x1;
    double r = 1.0;
    {
        KernelScope ks(*this, "polar_rotation");
        polar_scale_kernel<<<1, 256, 0, stream_>>>(a_dev, (int)n, fro2);
        polar_init_kernel<<<(count + 255) / 256, 256, 0, stream_>>>(a_dev, (int)n, fro2, cur);
        count_launch(2);
        for (int s0 = 0; s0 < max_steps && !(r < 1e-11); s0 += batch) {
            for (int s = 0; s < batch; ++s) {
                VQB_CUDA_CHECK(cudaMemsetAsync(resid, 0, sizeof(unsigned long long), stream_));
                polar_gram_kernel<<<grid, POLAR_TILE * POLAR_TILE, 0, stream_>>>(cur, (int)n, b, resid);
                polar_update_kernel<<<grid, POLAR_TILE * POLAR_TILE, 0, stream_>>>(cur, b, (int)n, resid, nxt);
                count_launch(2);
                std::swap(cur, nxt);
            }
            // the residual of the current iterate; the host looks at it once per batch of steps
            VQB_CUDA_CHECK(cudaMemsetAsync(resid, 0, sizeof(unsigned long long), stream_));
            polar_gram_kernel<<<grid, POLAR_TILE * POLAR_TILE, 0, stream_>>>(cur, (int)n, b, resid);
            count_launch();
            unsigned long long bits = 0;
            download(&bits, resid, sizeof bits);
            std::memcpy(&r, &bits, sizeof r);
        }
        polar_finish_kernel<<<(count + 255) / 256, 256, 0, stream_>>>(cur, count, rot_dev);
        count_launch();
        VQB_CUDA_CHECK(cudaGetLastError());
    }
    release(x0), release(x1), release(b), release(fro2), release(resid);
    return r < 1e-11;
}

} // namespace vqb
