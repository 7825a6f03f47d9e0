// Device-pointer entry points of the k-means trainer shared with the IVF index.
#pragma once

#include "common.cuh"
#include "tc_gemm.cuh"

namespace vb200 {

struct KMeansWorkspace {
    DevBuf<float> c_sq;     // |c_j|^2
    DevBuf<float> best;     // best score per point
    DevBuf<int32_t> counts; // k
    // centroid update in a fixed order: rows sorted by (label, row), the first row of each cluster
    DevBuf<uint32_t> sort_keys_in, sort_keys_out, sort_rows_in, sort_rows_out, cluster_off;
    DevBuf<uint8_t> sort_tmp;
    DevBuf<double> err;     // 1
    // tensor-core path: tiled bf16 terms of the points (kept while the same rows are assigned
    // again, i.e. across Lloyd iterations) and of the centroids, candidates, kernel scratch
    DevBuf<uint16_t> x_hi, x_lo, c_hi, c_lo;
    // nominations work on rows and centroids minus `shift`, scaled by `scale`, as fp16 terms (kmeans_assign_tc)
    DevBuf<float> shift, c_shifted, cs_sq;
    float scale = 0.f;
    bool half_off = false;        // too many rows were undecided that way: split bf16 terms from now on
    DevBuf<float> x_norm, xs_norm;   // |x_i| and |x_i - shift|, rounded up
    DevBuf<float> extremes;       // [0] largest |element| of the shifted rows and centroids, [1] max |c - shift|, [2] max |c|
    DevBuf<float> row_margin;     // twice the largest error of a row's scores
    DevBuf<float> x_sq;           // |x_i|^2, for the mean error
    DevBuf<uint32_t> close_rows;  // [0] how many, then the rows with several candidates within the margin
    DevBuf<unsigned long long> flagged_keys;
    DevBuf<float> row_bound;  // score of each row against its previous centroid (warm start)
    // rows whose tensor-core candidate lists may have lost a column (flagged by the kernel) are decided by
    // the fixed-order kernel over all centroids
    DevBuf<uint32_t> row_flags, flagged_rows, flagged_count;
    DevBuf<float> flagged_x, flagged_best;   // (many of them)
    DevBuf<int32_t> flagged_labels;
    const float* tiled_rows = nullptr;
    uint64_t tiled_n = 0;
    uint32_t tiled_dim = 0;
    DevBuf<uint64_t> cand;
    TcWorkspace tc;
    void
    forget_points() {
        tiled_rows = nullptr;
        tiled_n = 0;
        half_off = false;
    }
};

// True unless the environment variable VB200_DISABLE_TC is set to a non-zero value: the
// tensor-core candidate kernels are the default, the fixed-order SIMT kernels the cross-check.
bool tensor_cores_enabled();

// k-means++ seeding on the device; see vb200_kmeans_init.  picked_dev may be null.
int kmeans_pp_init_device(const float* x_dev, uint64_t n, uint32_t dim, uint32_t k, uint32_t seed,
                          float* centroids_dev, int64_t* picked_dev);

// labels_dev[i] = argmin_j |c_j|^2 - 2 <c_j, x_i> (lowest j on ties).  mean_err_host optional.
// prev_labels_dev (optional, may alias labels_dev): the labels of the previous Lloyd iteration; the
// tensor-core path uses them to skip centroids that cannot beat a row's previous one.
int kmeans_assign_device(KMeansWorkspace& ws, const float* x_dev, uint64_t n, uint32_t dim,
                         const float* centroids_dev, uint32_t k, int32_t* labels_dev,
                         double* mean_err_host, const int32_t* prev_labels_dev = nullptr);

// centroids_dev <- per-cluster means; empty clusters take row (j * 2654435761 + iter) % n.
int kmeans_update_device(KMeansWorkspace& ws, const float* x_dev, uint64_t n, uint32_t dim,
                         const int32_t* labels_dev, uint32_t k, uint32_t iter, float* centroids_dev);

}  // namespace vb200
