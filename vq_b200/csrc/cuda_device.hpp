// cuda_device.hpp -- the sm_100a implementation of vqb::Device plus the element-wise quantizers.
#pragma once
#include <cuda_runtime.h>

#include <atomic>
#include <map>
#include <memory>
#include <string>
#include <vector>

#include "backend.hpp"
#include "dense_tc.hpp"
#include "iter_status.cuh"
#include "pq_tc.hpp"

namespace vqb {

#define VQB_CUDA_CHECK(expr)                                                                                       \
    do {                                                                                                           \
        cudaError_t _e = (expr);                                                                                   \
        if (_e != cudaSuccess)                                                                                     \
            throw ::vqb::Error(100, std::string("CUDA error: ") + cudaGetErrorString(_e) + " at " + __FILE__ + ":" + \
                                        std::to_string(__LINE__));                                                 \
    } while (0)

class CudaDevice : public Device {
  public:
    explicit CudaDevice(int device);
    ~CudaDevice() override;

    void *alloc(size_t bytes) override;
    void *try_alloc(size_t bytes); // null when there is no room
    // Bytes of the buffer for the one-byte codes of a call (1M rows of 32 sub-spaces), which lives as long as the context.
    static constexpr size_t PQ_KEPT_CODES = size_t(32) << 20;
    uint8_t *pq_kept_codes() const { return pq_codes_; }
    void release(void *p) override;
    void upload(void *dst, const void *src, size_t bytes) override;
    void upload_queued(void *dst, const void *src, size_t bytes) override;
    void download(void *dst, const void *src, size_t bytes) override;
    // two of them with one wait (either may be empty)
    void download(void *dst, const void *src, size_t bytes, void *dst2, const void *src2, size_t bytes2);
    // The codebooks' operand of an encode with the same arguments, laid out before its rows are copied in; what it returns is the
    // operand_there of pq_encode_prepared.
    bool pq_encode_ahead(const Shape &sh, const float *x, const float *codebooks, int metric, const uint16_t *out_f16);
    void copy(void *dst, const void *src, size_t bytes) override;
    void zero(void *dst, size_t bytes) override;
    size_t code_bytes(size_t k) const override { return k <= 256 ? 1 : (k <= 65536 ? 2 : 4); }

    void prepare_rows(const Shape &sh, const float *x) override;
    size_t arriving_pieces(const float *x) override;
    size_t await_piece(const float *x, size_t piece) override;
    // Starts copying n rows of ld floats from the caller's host buffer to `dst` in pieces on a helper stream and remembers
    // them as arriving (Device::arriving_pieces).  Returns false, having copied nothing, when the rows are too few for pieces
    // to pay.  end_arrival waits (on the host) for whatever nobody has awaited yet; the owner of `dst` calls it before it
    // lets go of the memory or returns to the caller.
    bool begin_arrival(float *dst, const float *host, size_t n, size_t ld);
    void end_arrival();
    bool svd_sweeps(double *gt, double *vt, size_t n) override;
    bool polar_rotation(const double *a_dev, size_t n, float *rot_dev) override;
    void patch_centroids(const Shape &sh, const float *x, uint64_t row_begin, const RowPatch *patches, size_t n_patches,
                         float *centroids, Comm *comm) override;
    void assign_train(const Shape &sh, const float *x, const float *centroids, void *codes, const uint32_t *active,
                      const IterBuffers &buf) override;
    void accumulate(const Shape &sh, const float *x, const void *codes, const uint32_t *active, bool ordered,
                    const IterBuffers &buf) override;
    bool accumulate_moved(const Shape &sh, const float *x, void *codes_prev, const void *codes, const uint32_t *active,
                          const IterBuffers &local) override;
    void update_centroids(const Shape &sh, const IterBuffers &buf, const uint32_t *active, float *centroids,
                          IterStatus &status, const PeerExchange *px = nullptr) override;
    void rvq_update(float *res, size_t n, size_t dim, const float *centroids, size_t k, int metric, double p,
                    double *norm_sum) override;
    void pq_encode(const Shape &sh, const float *x, const float *codebooks, int metric, double p, uint16_t *out_f16,
                   uint32_t *out_codes, float *out_f32) override;
    void pq_encode_prepared(const Shape &sh, const float *x, const float *codebooks, int metric, double p, uint16_t *out_f16,
                            uint32_t *out_codes, bool operand_there);
    // The same encode on the CUDA-core kernels only: they work out of shared memory and registers and need no device
    // memory besides inputs and outputs.  Results are identical to pq_encode.
    void pq_encode_no_scratch(const Shape &sh, const float *x, const float *codebooks, int metric, double p, uint16_t *out_f16,
                              uint32_t *out_codes);
    void rotate_rows(const float *rot, size_t dim, const float *x, size_t n, float *y) override;
    bool encode_cross_cov(const Shape &sh, const float *x, const float *codebooks, int metric, double *a) override;
    void cross_cov(const float *y, const float *x, size_t n, size_t dim, double *a) override;

    // Not part of the training loops:
    void rvq_quantize(const float *x, size_t n, size_t dim, const float *codebooks, size_t stages, size_t k,
                      float epsilon, int metric, double p, uint16_t *out_f16, uint32_t *out_codes);
    // Raw scores, codes and the number of pairs left to the exact scan of the product-quantizer tensor-core kernel.
    void pq_tensor_debug(const float *x, size_t n, size_t m, const float *codebooks, size_t k, float *scores, uint32_t *codes,
                         unsigned long long *marked);
    // The fixed-point scores T of that kernel, the rows' sigma and K0, the sub-spaces' constants.
    void pq_fixed_point_debug(const float *x, size_t n, size_t m, size_t sd, const float *codebooks, size_t k, int metric, float *t, float *frames,
                              float *consts);
    // Reconstruction error and windowed recall@k of an f16 reconstruction (the reference's evaluation metrics).
    void evaluate_f16(const float *x, const uint16_t *q, size_t n, size_t dim, size_t k, float *mse_out, float *recall_out);
    void distance_rows(int metric, double p, const float *a, const float *b, size_t d, size_t n, float *out);
    void sq_quantize(float mn, float mx, size_t levels, float step, const float *x, size_t n, uint8_t *out);
    void bq_quantize(float threshold, uint8_t low, uint8_t high, const float *x, size_t n, uint8_t *out);

    // Two helper streams for overlapping host<->device copies with kernels (created on first use).
    cudaStream_t aux_stream(int i);
    void set_stream(cudaStream_t s); // nullptr = the CUDA default stream
    void reset_stream() { set_stream(own_stream_); }
    cudaStream_t stream() const { return stream_; }
    void synchronize();
    int device() const { return device_; }
    int sm_count() const { return sm_count_; }
    size_t smem_limit() const { return smem_limit_; }
    void end_call(); // at the end of every call of the C ABI
    int *error_word() const { return tc_error_; } // null with VQB_NO_TENSOR=1
    uint64_t launches() const { return launches_.load(); }
    void count_launch(uint64_t n = 1) { launches_ += n, unfinished_ = true; }
    // How often this context has asked CUDA for device or pinned memory (cudaMalloc, cudaMallocAsync, cudaHostAlloc).
    uint64_t device_allocs() const { return device_allocs_.load(); }
    void make_current() const;
    // Optional per-kernel timing with CUDA events on the launching stream (off by default).
    void set_timing(bool on);
    bool timing() const { return timing_; }
    void note_kernel(const char *name) { last_kernel_ = name; }
    void timing_begin(const char *name);
    void timing_end();
    // {"name": {"launches": L, "ms": T}, ...}; clears the record.
    std::string timing_report();
    // Diagnostic: raw tensor-core dot products (n x 256) and shortlist statistics {rows, candidates, full scans}.
    void dense_debug(const float *x, size_t n, size_t dim, const float *codebook, size_t k, float *dots, unsigned long long *stats3);
    // True when p points to device memory usable by kernels on this GPU.
    bool is_device_pointer(const void *p) const;

  private:
    int device_;
    int sm_count_ = 148;
    size_t smem_limit_ = 0;
    cudaStream_t own_stream_ = nullptr, stream_ = nullptr, aux_[2] = {nullptr, nullptr};
    // A call may leave work behind on its stream that uses the context's scratch, and the next call may run on another one: set_stream
    // puts that one behind order_event_.
    bool unfinished_ = false; // nothing has waited for stream_ since the last launch or copy
    cudaEvent_t order_event_ = nullptr;
    bool lasting(cudaStream_t s) const;
    static constexpr size_t STAGE_BYTES = 1u << 20; // pinned staging for small downloads
    static constexpr size_t UPLOAD_BYTES = 1u << 20; // behind it, a ring for small uploads
    size_t upload_at_ = 0;
    cudaEvent_t upload_event_ = nullptr; // the last of them has been read
    unsigned char *stage_ = nullptr, *stage_dev_ = nullptr; // stage_dev_: the same bytes as kernels on this GPU address them
    cudaEvent_t stage_event_ = nullptr;
    std::atomic<uint64_t> launches_{0}, device_allocs_{0};
    // page of mapped pinned memory the centroid-update kernels report to (iter_status.cuh)
    unsigned long long *status_host_ = nullptr, *status_dev_ = nullptr;
    size_t status_cap_words_ = 0;
    uint32_t status_seq_ = 0;
    StatusPage status_page(size_t m, size_t k);
    void wait_status(const StatusPage &sp, size_t m, size_t k, IterStatus &out);
    // centroids whose operand B (pq_tc.cu) the scratch currently holds, written by the fused centroid update
    const float *bop_fresh_ = nullptr;
    const float *dense_fresh_ = nullptr; // and those whose images (dense_tc.cu) dense_ holds, in its present frame
    // full-width tensor path (dense_tc.cu): which rows dense_ holds the images of, and the block behind dense_
    bool tensor_enabled_ = true;
    const float *prepared_x_ = nullptr;
    size_t prepared_n_ = 0, prepared_dim_ = 0;
    bool prepared_by_apply_ = false; // by rvq_update, for the k-means of the next stage
    DenseWork dense_;
    void *dense_block_ = nullptr;
    size_t dense_rows_ = 0, dense_for_ = 0, dense_dimp_ = 0; // rows it has room for, rows it was asked for
    // At most n rows at a time (dense_rows_; a multiple of 128 when fewer); `beside`: bytes a row that the caller allocates next.
    const DenseWork &dense_work(size_t n, size_t dim, size_t beside);
    void release_dense();
    void dense_decide(const float *x, size_t n, size_t dim, const float *codebook, size_t k, bool euclid, uint8_t *codes, uint32_t *changed,
                      unsigned long long *stats);
    float *pq_scratch_ = nullptr;
    std::unique_ptr<PqTcMaps> pq_maps_; // of pq_scratch_
    uint8_t *pq_codes_ = nullptr;       // PQ_KEPT_CODES bytes
    float *rot_split_ = nullptr; // TF32 high and low parts of the rotation matrix of the current rotate_rows call (dim <= 128)
    bool opq_tensor_enabled_ = true;
    bool pq_tensor_enabled_ = false;
    unsigned long long *tc_stats_ = nullptr;
    int *tc_error_ = nullptr;
    void ensure_tc_buffers();
    void pq_encode_impl(const Shape &sh, const float *x, const float *codebooks, int metric, double p, uint16_t *out_f16,
                        uint32_t *out_codes, float *out_f32, bool cuda_cores_only, bool operand_there);

    void check_tc_error();
    // rows on their way from a host buffer (begin_arrival): piece i is complete when arrival_done_[i] has fired
    struct Arrival {
        const float *dev = nullptr, *host = nullptr;
        size_t n = 0, ld = 0, piece_rows = 0, pieces = 0, awaited = 0;
    } arrival_;
    std::vector<cudaEvent_t> arrival_done_; // created once, re-used
    cudaEvent_t arrival_fence_ = nullptr;
    bool timing_ = false;
    const char *last_kernel_ = "(none)"; // for the message of a wait that was given up
    struct Span {
        const char *name;
        cudaEvent_t a, b;
    };
    std::vector<Span> spans_;
    std::vector<cudaEvent_t> event_pool_; // timing events are created once and re-used
    cudaEvent_t take_event();
};

// Brackets one kernel launch for the optional timing record.
struct KernelScope {
    CudaDevice &dev;
    KernelScope(CudaDevice &d, const char *name) : dev(d)
    {
        dev.note_kernel(name);
        if (dev.timing()) dev.timing_begin(name);
    }
    ~KernelScope()
    {
        if (dev.timing()) dev.timing_end();
    }
};

// Lets a kernel be launched with all the dynamic shared memory that there is beside its own arrays.  Always the same figure, set once: the attribute
// is the kernel's and not the launch's, so that a thread that sets what its own launch needs takes it away from another one's (two contexts,
// fits with different numbers of centroids) between that one's call and launch.
void allow_shared_memory(const CudaDevice &dev, const void *kernel);
template <typename... P> void allow_shared_memory(const CudaDevice &dev, void (*kernel)(P...)) { allow_shared_memory(dev, reinterpret_cast<const void *>(kernel)); }

// As launch_following (below), in clusters of CTAs along x.
template <typename... P, typename... A>
void launch_following_clusters(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, unsigned cluster, cudaStream_t stream, A &&...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid, cfg.blockDim = block, cfg.dynamicSmemBytes = smem, cfg.stream = stream;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster, attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = cluster > 1 ? 2 : 1;
    VQB_CUDA_CHECK(cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...));
}

// Launches a kernel that may start while the one before it in the stream still runs: it waits itself (after_previous_kernel() of
// kernels_common.cuh, before its first access to global memory), so that its launch and set-up overlap the other's end.  Between two
// small kernels that takes 1 to 3 us off: encode of 3000 / 20,000 x 128 (three kernels) 20.9 -> 15.5 / 28.4 -> 24.1 us, fit of 2500 /
// 10,000 x 128 (five kernels an iteration) 587 -> 507 / 599 -> 540 us; residual fit (3 stages) of 3000 x 64 / 20,000 x 128 1830 -> 1495 /
// 2440 -> 2220 us; tree of 100,000 x 128 1387 -> 1320 us.
template <typename... P, typename... A>
void launch_following(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A &&...args)
{
    launch_following_clusters(kernel, grid, block, smem, 1, stream, static_cast<A &&>(args)...);
}

// assign_launch.cu
struct AssignParams;
struct GenericParams;
// Returns false when the register kernel does not cover this shape/metric.
bool launch_assign_reg(CudaDevice &dev, const AssignParams &p, int metric, bool train, size_t code_bytes);
void launch_assign_generic(CudaDevice &dev, GenericParams &p, int metric, int mode, size_t code_bytes);

} // namespace vqb
