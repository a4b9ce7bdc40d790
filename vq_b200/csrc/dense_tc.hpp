// dense_tc.hpp -- full-width nearest-centroid search: tensor-core shortlist (dense_tc.cu), exact decision and what follows it in
// the residual quantizer (resolve.cu).
#pragma once
#include <cstddef>
#include <cstdint>

namespace vqb {

class CudaDevice;

#define DENSE_MASK_WORDS 8 /* 256 candidate bits per row (32 bytes) */
#define VQB_DENSE_INF __int_as_float(0x7f800000)

// Squared-Euclidean / Euclidean, 16 < dim <= 128, 2 <= k <= 256.  (Narrower rows fill a fraction of a K step and of a line;
// the register kernels serve them.)
bool dense_tc_applicable(size_t dim, size_t k, int metric);
size_t dense_tc_smem_bytes();
// a row's image is 2 * dense_padded(dim) binary16 values (dense_image.cuh)
inline size_t dense_padded(size_t dim) { return (dim + 15) / 16 * 16; }

// Device memory of one fit or encode, for up to a given number of rows.
struct DenseWork {
    uint16_t *image = nullptr;      // [n][2 * dense_padded(dim)]
    float *norms = nullptr;         // [n] upper bounds of |s (x - mu)|^2
    uint32_t *cand = nullptr;       // [n][8] bit j set: centroid j may be the reference's choice (all k bits set: examine all)
    uint32_t *list = nullptr;       // [n] rows with more than one candidate
    uint32_t *list_count = nullptr; // [3] how many, CTAs that are done with them (both zero between passes), how many the last pass had
    uint16_t *book_image = nullptr; // [256][2 * dense_padded(dim)]
    float *half_norms = nullptr;    // [256]
    float *frame = nullptr;         // [129] mu and s (dense_image.cuh)
};

// w.frame for these rows, or (codes != null) for their residuals x - centroid; center = false: mu = 0
void dense_frame(CudaDevice &dev, const DenseWork &w, const float *x, size_t n, size_t dim, const float *codebook, const uint8_t *codes, bool center);
// image and norms of the rows in w.frame
void dense_prepare(CudaDevice &dev, const DenseWork &w, const float *x, size_t n, size_t dim);

// Decides every row that has a single candidate -- codes[r] is rewritten, *changed gets VQB_MOVED_BITS when a row moved -- and
// appends the other rows (also those that cannot be ranked: NaN, infinity) to w.list with their masks in w.cand
// (*w.list_count zero on entry); book_there: w holds the codebook's image already.  Without `train` all rows get their mask and nothing else happens (diagnostics).
struct ShortlistTrain {
    uint8_t *codes;
    uint32_t *changed;
};
void dense_shortlist(CudaDevice &dev, const DenseWork &w, size_t n, size_t dim, const float *codebook, size_t k, unsigned long long *stats,
                     int *error_word, float *debug_dots, const ShortlistTrain *train, bool book_there);

// The listed rows: the reference's own arithmetic over their candidates.
void dense_resolve(CudaDevice &dev, const DenseWork &w, const float *x, size_t n, size_t dim, const float *codebook, size_t k, bool euclid,
                   uint8_t *codes, uint32_t *changed);

// One step of the residual quantizer after a row's code is known: res = x - centroid (x may be res), and the new rows' images
// and norms, in a new frame, for the next stage.
struct RvqApply {
    const float *x = nullptr;
    float *res = nullptr;
    size_t n = 0, dim = 0;
    const float *codebook = nullptr;
    const uint8_t *codes = nullptr;
    double *norm_sum = nullptr;  // the residual norms are added up (src/rvq.rs:131-138)
};
void rvq_apply(CudaDevice &dev, const RvqApply &a, const DenseWork &w);

// The residual encoder with all its stages in one kernel (rvq_tc.cu), for shapes that dense_tc_applicable takes.
struct GenericParams;
bool rvq_stages_pays(const GenericParams &g);                        // more rows than direct.cu is faster with
bool rvq_stages_one_launch(const GenericParams &g);                  // so few that the kernel lays the codebooks out itself
size_t rvq_stages_bytes(size_t dim, size_t k, size_t stages);        // device memory that it needs
void launch_rvq_stages(CudaDevice &dev, const GenericParams &g, bool euclid, void *work);

} // namespace vqb
