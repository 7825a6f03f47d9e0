// Exact BruteForce kNN over fp32 or bf16 rows: dense score slabs select a few candidates more
// than k per query, which are then re-scored in the reference's arithmetic and ordered.
#include <algorithm>
#include <cmath>
#include <vector>

#include "bf_stream.cuh"
#include "dense.cuh"
#include "kmeans.cuh"
#include "comm.cuh"
#include "tc_gemm.cuh"

namespace vb200 {

constexpr uint32_t BF_SLACK = 16;                 // candidates kept beyond k before re-scoring
constexpr double BF_MATRIX_SCORES = 4e8;          // scores of a batch that goes through a score matrix, at most
constexpr size_t BF_PINNED_BYTES = 256 * 1024;    // host results of a search that pass through pinned memory, at most
constexpr uint64_t BF_COL_CHUNK = uint64_t{1} << 20;
constexpr uint64_t BF_SLAB_FLOATS = uint64_t{256} << 20;  // 1 GiB of scores

// generic::FloatToBF16 (src/simd/generic.cpp:198-202): add 0x8000, keep the high half.
__global__ void
float_to_bf16_kernel(const float* __restrict__ in, uint64_t n, uint16_t* __restrict__ out) {
    uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) {
        out[i] = static_cast<uint16_t>((__float_as_uint(in[i]) + 0x8000u) >> 16);
    }
}

// One CTA per query, one thread per candidate: distance as the reference computes it for one
// row -- an FMA chain over the dimensions in ascending order
// (FP32Quantizer::ComputeDistImpl, src/quantization/fp32_quantizer.cpp:163-190;
// HalfPrecisionQuantizer, src/quantization/scalar_quantization/half_precision_quantizer.cpp:54-123)
// -- then a sort by (distance, row).
template <typename T>
__global__ void __launch_bounds__(128)
bf_rescore_kernel(const T* __restrict__ queries, uint32_t dim, const T* __restrict__ base,
                  const uint64_t* __restrict__ cand, uint32_t ncand, uint32_t n2, uint32_t k,
                  int metric, uint64_t* __restrict__ out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* keys = reinterpret_cast<uint64_t*>(smem_raw);
    float* qf = reinterpret_cast<float*>(keys + n2);   // the query, widened once
    const T* q = queries + static_cast<uint64_t>(blockIdx.x) * dim;
    const uint64_t* cq = cand + static_cast<uint64_t>(blockIdx.x) * ncand;
    for (uint32_t d = threadIdx.x; d < dim; d += blockDim.x) {
        qf[d] = widen(q[d]);
    }
    __syncthreads();
    constexpr uint32_t VEC = 16 / sizeof(T);           // elements per 16-byte load
    const bool wide_loads = dim % VEC == 0 && (reinterpret_cast<uintptr_t>(base) & 15u) == 0;
    for (uint32_t i = threadIdx.x; i < n2; i += blockDim.x) {
        uint64_t key = KEY_INF;
        // candidates with an infinite nominating score are filtered-out rows that only filled up a
        // short list: they are not results
        if (i < ncand && cq[i] != KEY_INF && static_cast<uint32_t>(cq[i] >> 32) < 0xFF800000u) {
            uint32_t row = static_cast<uint32_t>(cq[i]);
            const T* x = base + static_cast<uint64_t>(row) * dim;
            float s = 0.f;
            const bool l2 = metric == VB200_METRIC_L2;
            if (wide_loads) {
                // same chain, rows fetched sixteen bytes at a time with a few loads in flight
                const uint4* xv = reinterpret_cast<const uint4*>(x);
                const uint32_t nv = dim / VEC;
                for (uint32_t v0 = 0; v0 < nv; v0 += 4) {
                    uint4 w[4];
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u) {
                        w[u] = v0 + u < nv ? __ldg(xv + v0 + u) : make_uint4(0, 0, 0, 0);
                    }
#pragma unroll
                    for (uint32_t u = 0; u < 4; ++u) {
                        if (v0 + u < nv) {
                            T e[VEC];
                            *reinterpret_cast<uint4*>(e) = w[u];
                            const float* qq = qf + (v0 + u) * VEC;
#pragma unroll
                            for (uint32_t j = 0; j < VEC; ++j) {
                                if (l2) {
                                    float t = __fsub_rn(widen(e[j]), qq[j]);
                                    s = fmaf(t, t, s);
                                } else {
                                    s = fmaf(widen(e[j]), qq[j], s);
                                }
                            }
                        }
                    }
                }
            } else if (l2) {
                for (uint32_t d = 0; d < dim; ++d) {
                    float t = __fsub_rn(widen(x[d]), qf[d]);
                    s = fmaf(t, t, s);
                }
            } else {
                for (uint32_t d = 0; d < dim; ++d) {
                    s = fmaf(widen(x[d]), qf[d], s);
                }
            }
            if (!l2) {
                s = __fsub_rn(1.0f, s);
            }
            key = make_key(s, row);
        }
        keys[i] = key;
    }
    block_bitonic_sort(keys, n2);
    uint64_t* dst = out + static_cast<uint64_t>(blockIdx.x) * k;
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
        dst[i] = i < n2 ? keys[i] : KEY_INF;
    }
}

template <typename T>
static int
bf_rescore(const T* queries, uint64_t nq, uint32_t dim, const T* base, const uint64_t* cand, uint32_t ncand, uint32_t n2,
           uint32_t k, int metric, uint64_t* out) {
    const size_t smem = n2 * sizeof(uint64_t) + dim * sizeof(float);
    VB_CHECK_ARG(smem <= 200 * 1024, "dim = %u is too large for the exact re-scoring step", dim);
    auto kernel = bf_rescore_kernel<T>;
    VB_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem));
    VB_LAUNCH(kernel, static_cast<uint32_t>(nq), 128, smem, queries, dim, base, cand, ncand, n2, k, metric, out);
    return 0;
}

// One block per query: the k best keys of its `per_query` partial keys and, when `prev` is given, of the k
// keys an earlier call left there (prev may be `out`).  bound_out[q], when asked for, is the score of the
// k-th key found, or +inf while fewer than k exist: no key scoring at or above it can enter the k best later.
__global__ void __launch_bounds__(256)
bf_merge_kernel(const uint64_t* __restrict__ part, uint64_t per_query, const uint64_t* prev, uint32_t k, uint32_t cap,
                uint64_t* out, float* __restrict__ bound_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    uint64_t* keys = reinterpret_cast<uint64_t*>(smem_raw);
    uint32_t* state = reinterpret_cast<uint32_t*>(keys + cap);
    BlockSelect sel;
    sel.init(keys, state, k, cap);
    const uint64_t* src = part + static_cast<uint64_t>(blockIdx.x) * per_query;
    const uint64_t n_prev = prev != nullptr ? k : 0;
    const uint64_t* old = prev != nullptr ? prev + static_cast<uint64_t>(blockIdx.x) * k : nullptr;
    for (uint64_t base = 0; base < per_query + n_prev; base += blockDim.x) {
        sel.make_room(blockDim.x);
        uint64_t thr = sel.threshold();
        uint64_t i = base + threadIdx.x;
        if (i < per_query + n_prev) {
            uint64_t key = i < n_prev ? old[i] : __ldg(src + (i - n_prev));
            if (key != KEY_INF) {
                sel.offer(key, thr);
            }
        }
    }
    uint32_t cnt = sel.finish();
    uint64_t* dst = out + static_cast<uint64_t>(blockIdx.x) * k;
    for (uint32_t i = threadIdx.x; i < k; i += blockDim.x) {
        dst[i] = i < cnt ? keys[i] : KEY_INF;
    }
    if (bound_out != nullptr && threadIdx.x == 0) {
        bound_out[blockIdx.x] = cnt >= k ? ordered_to_float(static_cast<uint32_t>(keys[k - 1] >> 32)) : INFINITY;
    }
}

__global__ void
bf_results_kernel(const uint64_t* __restrict__ keys, uint64_t total, const int64_t* __restrict__ labels,
                  int64_t* __restrict__ ids, float* __restrict__ dists, uint64_t* __restrict__ keys_out) {
    uint64_t e = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e >= total) {
        return;
    }
    uint64_t key = keys[e];
    if (keys_out != nullptr) {
        keys_out[e] = key;
    }
    if (key == KEY_INF) {
        ids[e] = -1;
        if (dists != nullptr) {
            dists[e] = INFINITY;
        }
    } else {
        ids[e] = labels[static_cast<uint32_t>(key)];
        if (dists != nullptr) {
            dists[e] = ordered_to_float(static_cast<uint32_t>(key >> 32));
        }
    }
}

// bias[i] = the row's score bias (its squared norm for L2, 0 for IP), or +inf when row i is
// removed or filtered out: an infinite score is never nominated.
__global__ void
bf_masked_bias_kernel(const float* __restrict__ norms, uint64_t n, const uint32_t* __restrict__ tomb,
                      const uint32_t* __restrict__ deny, uint64_t deny_bits, const int64_t* __restrict__ labels,
                      const uint64_t* __restrict__ label_bits, uint64_t n_label_bits, float* __restrict__ bias) {
    uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) {
        return;
    }
    bool out = tomb != nullptr && ((tomb[i >> 5] >> (i & 31u)) & 1u);
    if (!out && deny != nullptr && i < deny_bits) {
        out = (deny[i >> 5] >> (i & 31u)) & 1u;
    }
    if (!out && label_bits != nullptr) {
        const uint64_t bit = static_cast<uint64_t>(labels[i]) & 0xFFFFFFFFull;
        out = bit < n_label_bits && ((label_bits[bit >> 6] >> (bit & 63u)) & 1ull);
    }
    bias[i] = out ? INFINITY : (norms != nullptr ? norms[i] : 0.f);
}

__global__ void
bf_tombstone_kernel(const int64_t* __restrict__ labels, uint64_t n, const int64_t* __restrict__ sorted, uint64_t count,
                    uint32_t* __restrict__ tomb, unsigned long long* __restrict__ newly) {
    uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) {
        return;
    }
    const int64_t label = labels[i];
    uint64_t lo = 0, hi = count;
    while (lo < hi) {
        const uint64_t mid = (lo + hi) >> 1;
        if (sorted[mid] < label) {
            lo = mid + 1;
        } else {
            hi = mid;
        }
    }
    if (lo < count && sorted[lo] == label) {
        const uint32_t bit = 1u << (i & 31u);
        if ((atomicOr(tomb + (i >> 5), bit) & bit) == 0u) {
            atomicAdd(newly, 1ull);
        }
    }
}

}  // namespace vb200

using namespace vb200;

struct vb200_bf {
    uint32_t dim = 0;
    int metric = 0, quant = 0;
    // cosine: rows and queries are normalised, then it is the inner-product index
    // (FP32Quantizer / HalfPrecisionQuantizer with METRIC_TYPE_COSINE)
    bool cosine = false;
    DevBuf<float> q_unit;
    // removed rows (MARK_REMOVE) and the id filter of the running search
    DevBuf<uint32_t> tombstones;
    uint64_t tomb_words = 0, n_removed = 0;
    const vb200_filter* filter = nullptr;
    DevBuf<float> masked_bias;
    uint64_t n = 0;
    DevBuf<float> base_f32;
    DevBuf<uint16_t> base_bf16;
    DevBuf<float> norms;
    DevBuf<int64_t> labels;
    // search workspace
    DevBuf<float> q_f32, scores;
    DevBuf<uint16_t> q_bf16;
    DevBuf<uint64_t> part, cand, keys;
    // tensor-core path: the base (and per search the queries) as tiled bf16 terms
    DevBuf<uint16_t> base_hi, base_lo, q_hi, q_lo;
    bool tiled_valid = false;
    // of the tiled rows, one of every sample_stride (0: none taken yet) with its score bias, see bf_take_sample
    DevBuf<uint16_t> sample_hi, sample_lo;
    DevBuf<float> sample_bias;
    uint32_t sample_stride = 0;
    DevBuf<uint64_t> tc_out;
    DevBuf<uint32_t> list_count;   // entries of every list of tc_out
    DevBuf<uint64_t> spill;        // entries of a query that its lists have no room for, with their number
    DevBuf<uint32_t> spilled;
    DevBuf<uint64_t> sh_local, sh_all;   // sharded search: this rank's packed [keys | labels] and the gathered ones
    DevBuf<float> row_bound;   // per query: the kcand-th candidate score after the column ranges searched so far
    TcWorkspace tc;
    DevBuf<int64_t> out_ids;
    DevBuf<float> out_dists;
    DevBuf<uint32_t> stream_bound;   // per query: a bound of its k-th best distance while rows stream by
    DevBuf<float> row_max;           // the largest norm of a row
    // a batch's score matrix: [0] the kernel's error flag, [1] how many queries' nominations may not have been enough, then which
    DevBuf<uint32_t> unsure;
    PinnedBuf pinned;                // small host inputs and results
    std::mutex mu;
};

template <typename T>
static int
bf_grow(DevBuf<T>& buf, size_t keep, size_t need) {
    if (need <= buf.cap) {
        return 0;
    }
    size_t cap = buf.cap * 2 > need ? buf.cap * 2 : need;
    DevBuf<T> bigger;
    if (bigger.reserve(cap) != 0) {
        VB_TRY(bigger.reserve(need));
    }
    if (keep > 0) {
        VB_CUDA(cudaMemcpyAsync(bigger.ptr, buf.ptr, keep * sizeof(T), cudaMemcpyDeviceToDevice,
                                current_stream()));
        VB_TRY(sync_stream());
    }
    buf = std::move(bigger);
    return 0;
}

extern "C" int
vb200_bf_create(uint32_t dim, int metric, int quant, vb200_bf_t* out) {
    VB_CHECK_ARG(out != nullptr, "null output handle");
    VB_CHECK_ARG(dim > 0, "dim must be positive");
    VB_CHECK_ARG(metric == VB200_METRIC_L2 || metric == VB200_METRIC_IP || metric == VB200_METRIC_COSINE,
                 "metric_type must be l2, ip or cosine (got %d)", metric);
    VB_CHECK_ARG(quant == VB200_QUANT_FP32 || quant == VB200_QUANT_BF16,
                 "base_quantization_type must be fp32 or bf16 for this engine (got %d)", quant);
    if (vb200_device_count() <= 0) {
        VB_FAIL(VB200_INTERNAL_ERROR, "no CUDA device available; this engine has no CPU path");
    }
    vb200_bf* ix = new (std::nothrow) vb200_bf();
    if (ix == nullptr) {
        VB_FAIL(VB200_NO_ENOUGH_MEMORY, "out of host memory");
    }
    ix->dim = dim;
    ix->metric = metric == VB200_METRIC_COSINE ? VB200_METRIC_IP : metric;
    ix->cosine = metric == VB200_METRIC_COSINE;
    ix->quant = quant;
    *out = ix;
    return 0;
}

extern "C" int
vb200_bf_destroy(vb200_bf_t ix) {
    if (ix == nullptr) {
        return 0;
    }
    ReleaseScope scope;
    delete ix;
    return 0;
}

static int
bf_append_labels_and_norms(vb200_bf* ix, const int64_t* ids, uint64_t count) {
    VB_TRY(bf_grow(ix->labels, ix->n, ix->n + count));
    VB_CUDA(cudaMemcpyAsync(ix->labels.ptr + ix->n, ids, count * sizeof(int64_t), cudaMemcpyDefault,
                            current_stream()));
    VB_TRY(bf_grow(ix->norms, ix->n, ix->n + count));
    if (ix->quant == VB200_QUANT_FP32) {
        VB_TRY(row_sqnorm_f32(ix->base_f32.ptr + ix->n * ix->dim, count, ix->dim, ix->norms.ptr + ix->n));
    } else {
        VB_TRY(row_sqnorm_bf16(ix->base_bf16.ptr + ix->n * ix->dim, count, ix->dim, ix->norms.ptr + ix->n));
    }
    if (ix->row_max.ptr == nullptr) {
        VB_TRY(ix->row_max.reserve(1));
        VB_CUDA(cudaMemsetAsync(ix->row_max.ptr, 0, sizeof(float), current_stream()));
    }
    VB_LAUNCH(bf_row_max_kernel, static_cast<uint32_t>(std::min<uint64_t>((count + 1023) / 1024, 4ull * sm_count())), 256, 0,
              ix->norms.ptr + ix->n, count, ix->row_max.ptr);
    {
        // tombstone words for the new rows
        const uint64_t words = (ix->n + count + 31) / 32;
        if (words > ix->tomb_words) {
            DevBuf<uint32_t> bigger;
            const uint64_t cap = words * 2;
            VB_TRY(bigger.reserve(cap));
            VB_CUDA(cudaMemsetAsync(bigger.ptr, 0, cap * sizeof(uint32_t), current_stream()));
            if (ix->tomb_words > 0) {
                VB_CUDA(cudaMemcpyAsync(bigger.ptr, ix->tombstones.ptr, ix->tomb_words * sizeof(uint32_t),
                                        cudaMemcpyDeviceToDevice, current_stream()));
            }
            VB_TRY(sync_stream());
            ix->tombstones = std::move(bigger);
            ix->tomb_words = cap;
        }
    }
    VB_TRY(sync_stream());
    ix->n += count;
    ix->tiled_valid = false;
    return 0;
}

extern "C" int
vb200_bf_add(vb200_bf_t ix, const float* data, uint64_t count, const int64_t* ids) {
    VB_CHECK_ARG(ix != nullptr, "null index");
    if (count == 0) {
        return 0;
    }
    VB_CHECK_ARG(data != nullptr && ids != nullptr, "null pointer");
    std::lock_guard<std::mutex> lock(ix->mu);
    VB_CHECK_ARG(ix->n + count < 0xFFFFFFFFull, "index would exceed 2^32-1 vectors");
    const uint64_t elems = count * ix->dim;
    if (ix->quant == VB200_QUANT_FP32 && !ix->cosine) {
        VB_TRY(bf_grow(ix->base_f32, ix->n * ix->dim, (ix->n + count) * ix->dim));
        VB_CUDA(cudaMemcpyAsync(ix->base_f32.ptr + ix->n * ix->dim, data, elems * sizeof(float),
                                cudaMemcpyDefault, current_stream()));
    } else {
        DevInput<float> x;
        VB_TRY(x.bind(data, elems));
        DevBuf<float> unit_rows;
        const float* xr = x.ptr;
        if (ix->quant == VB200_QUANT_FP32) {
            VB_TRY(bf_grow(ix->base_f32, ix->n * ix->dim, (ix->n + count) * ix->dim));
            VB_TRY(normalize_rows_f32(x.ptr, count, ix->dim, ix->base_f32.ptr + ix->n * ix->dim));
        } else {
            if (ix->cosine) {
                VB_TRY(unit_rows.reserve(elems));
                VB_TRY(normalize_rows_f32(x.ptr, count, ix->dim, unit_rows.ptr));
                xr = unit_rows.ptr;
            }
            VB_TRY(bf_grow(ix->base_bf16, ix->n * ix->dim, (ix->n + count) * ix->dim));
            uint64_t blocks = (elems + 255) / 256;
            VB_CHECK_ARG(blocks <= 0x7fffffffu, "add batch too large");
            VB_LAUNCH(float_to_bf16_kernel, static_cast<uint32_t>(blocks), 256, 0, xr, elems,
                      ix->base_bf16.ptr + ix->n * ix->dim);
        }
        VB_TRY(sync_stream());
    }
    return bf_append_labels_and_norms(ix, ids, count);
}

extern "C" int
vb200_bf_add_bf16(vb200_bf_t ix, const uint16_t* data, uint64_t count, const int64_t* ids) {
    VB_CHECK_ARG(ix != nullptr, "null index");
    if (count == 0) {
        return 0;
    }
    VB_CHECK_ARG(data != nullptr && ids != nullptr, "null pointer");
    VB_CHECK_ARG(ix->quant == VB200_QUANT_BF16, "index does not store bf16 rows");
    VB_CHECK_ARG(!ix->cosine, "a cosine index normalises fp32 rows before rounding them: add them with vb200_bf_add");
    std::lock_guard<std::mutex> lock(ix->mu);
    VB_CHECK_ARG(ix->n + count < 0xFFFFFFFFull, "index would exceed 2^32-1 vectors");
    VB_TRY(bf_grow(ix->base_bf16, ix->n * ix->dim, (ix->n + count) * ix->dim));
    VB_CUDA(cudaMemcpyAsync(ix->base_bf16.ptr + ix->n * ix->dim, data, count * ix->dim * sizeof(uint16_t),
                            cudaMemcpyDefault, current_stream()));
    return bf_append_labels_and_norms(ix, ids, count);
}

extern "C" int
vb200_bf_get_rows(vb200_bf_t ix, void* rows) {
    VB_CHECK_ARG(ix != nullptr && rows != nullptr, "null pointer");
    std::lock_guard<std::mutex> lock(ix->mu);
    if (ix->n == 0) {
        return 0;
    }
    const uint64_t elems = ix->n * ix->dim;
    if (ix->quant == VB200_QUANT_FP32) {
        VB_TRY(copy_out(static_cast<float*>(rows), ix->base_f32.ptr, elems));
    } else {
        VB_TRY(copy_out(static_cast<uint16_t*>(rows), ix->base_bf16.ptr, elems));
    }
    return sync_stream();
}

extern "C" int
vb200_bf_set_rows(vb200_bf_t ix, const void* rows, uint64_t count, const int64_t* ids) {
    VB_CHECK_ARG(ix != nullptr, "null index");
    std::lock_guard<std::mutex> lock(ix->mu);
    if (ix->n != 0) {
        VB_FAIL(VB200_WRONG_STATUS, "stored rows can only be loaded into an empty index");
    }
    if (count == 0) {
        return 0;
    }
    VB_CHECK_ARG(rows != nullptr && ids != nullptr, "null pointer");
    VB_CHECK_ARG(count < 0xFFFFFFFFull, "index would exceed 2^32-1 vectors");
    const uint64_t elems = count * ix->dim;
    if (ix->quant == VB200_QUANT_FP32) {
        VB_TRY(bf_grow(ix->base_f32, 0, elems));
        VB_CUDA(cudaMemcpyAsync(ix->base_f32.ptr, rows, elems * sizeof(float), cudaMemcpyDefault, current_stream()));
    } else {
        VB_TRY(bf_grow(ix->base_bf16, 0, elems));
        VB_CUDA(cudaMemcpyAsync(ix->base_bf16.ptr, rows, elems * sizeof(uint16_t), cudaMemcpyDefault,
                                current_stream()));
    }
    return bf_append_labels_and_norms(ix, ids, count);
}

extern "C" int64_t
vb200_bf_num_elements(vb200_bf_t ix) {
    return ix == nullptr ? 0 : static_cast<int64_t>(ix->n - ix->n_removed);
}

extern "C" int
vb200_bf_remove(vb200_bf_t ix, const int64_t* labels, uint64_t count, uint64_t* removed) {
    VB_CHECK_ARG(ix != nullptr, "null index");
    if (removed != nullptr) {
        *removed = 0;
    }
    if (count == 0) {
        return 0;
    }
    VB_CHECK_ARG(labels != nullptr, "null pointer");
    std::lock_guard<std::mutex> lock(ix->mu);
    if (ix->n == 0) {
        return 0;
    }
    std::vector<int64_t> sorted(count);
    VB_CUDA(cudaMemcpy(sorted.data(), labels, count * sizeof(int64_t), cudaMemcpyDefault));
    std::sort(sorted.begin(), sorted.end());
    DevBuf<int64_t> sorted_dev;
    DevBuf<unsigned long long> newly;
    VB_TRY(sorted_dev.reserve(count));
    VB_TRY(newly.reserve(1));
    cudaStream_t st = current_stream();
    VB_CUDA(cudaMemcpyAsync(sorted_dev.ptr, sorted.data(), count * sizeof(int64_t), cudaMemcpyHostToDevice, st));
    VB_CUDA(cudaMemsetAsync(newly.ptr, 0, sizeof(unsigned long long), st));
    VB_LAUNCH(bf_tombstone_kernel, static_cast<uint32_t>((ix->n + 255) / 256), 256, 0, ix->labels.ptr, ix->n,
              sorted_dev.ptr, count, ix->tombstones.ptr, newly.ptr);
    unsigned long long n_new = 0;
    VB_CUDA(cudaMemcpyAsync(&n_new, newly.ptr, sizeof(n_new), cudaMemcpyDeviceToHost, st));
    VB_TRY(sync_stream());
    ix->n_removed += n_new;
    if (removed != nullptr) {
        *removed = n_new;
    }
    return 0;
}

// The queries on the device and the rows' masks, as bf_stage leaves them.
struct BfStaged {
    const float *queries = nullptr, *bias = nullptr;
    bool masked = false;
};

// What every search starts with: the queries on the device (normalised for cosine, rounded for bf16 rows) and
// the score bias per row -- |x|^2 for L2, none for IP, +inf for rows that are removed or filtered out.
static int
bf_stage(vb200_bf* ix, const float* queries, uint64_t nq, BfStaged* out) {
    const uint32_t dim = ix->dim;
    const uint64_t n = ix->n;
    const float* q_dev = queries;
    if (!is_device_pointer(queries)) {
        VB_TRY(ix->q_f32.reserve(nq * dim));
        VB_CUDA(cudaMemcpyAsync(ix->q_f32.ptr, queries, nq * dim * sizeof(float), cudaMemcpyHostToDevice,
                                current_stream()));
        q_dev = ix->q_f32.ptr;
    }
    if (ix->cosine) {
        VB_TRY(ix->q_unit.reserve(nq * dim));
        VB_TRY(normalize_rows_f32(q_dev, nq, dim, ix->q_unit.ptr));
        q_dev = ix->q_unit.ptr;
    }
    if (ix->quant == VB200_QUANT_BF16) {
        VB_TRY(ix->q_bf16.reserve(nq * dim));
        VB_LAUNCH(float_to_bf16_kernel, static_cast<uint32_t>((nq * dim + 255) / 256), 256, 0, q_dev,
                  nq * dim, ix->q_bf16.ptr);
    }
    const float* bias_all = ix->metric == VB200_METRIC_L2 ? ix->norms.ptr : nullptr;
    const vb200_filter* f = ix->filter;
    const bool user_deny = f != nullptr && f->deny_inner_bits != nullptr && f->n_inner_bits > 0;
    const bool user_labels = f != nullptr && f->invalid_label_bits != nullptr && f->n_label_bits > 0;
    out->masked = ix->n_removed > 0 || user_deny || user_labels;
    if (out->masked) {
        DevInput<uint32_t> deny;
        DevInput<uint64_t> lbits;
        if (user_deny) {
            VB_TRY(deny.bind(f->deny_inner_bits, (f->n_inner_bits + 31) / 32));
        }
        if (user_labels) {
            VB_TRY(lbits.bind(f->invalid_label_bits, (f->n_label_bits + 63) / 64));
        }
        VB_TRY(ix->masked_bias.reserve(n));
        VB_LAUNCH(bf_masked_bias_kernel, static_cast<uint32_t>((n + 255) / 256), 256, 0, bias_all, n,
                  ix->n_removed > 0 ? ix->tombstones.ptr : nullptr, user_deny ? deny.ptr : nullptr,
                  user_deny ? f->n_inner_bits : 0, ix->labels.ptr, user_labels ? lbits.ptr : nullptr,
                  user_labels ? f->n_label_bits : 0, ix->masked_bias.ptr);
        VB_TRY(sync_stream());   // the staged bitmaps end with this scope
        bias_all = ix->masked_bias.ptr;
    }
    out->queries = q_dev;
    out->bias = bias_all;
    return 0;
}

// The rows as tiled bf16 terms for the tensor cores, made at the first search that needs them after an add.
static int
bf_tile_base(vb200_bf* ix) {
    if (ix->tiled_valid) {
        return 0;
    }
    const size_t elems = tc_tiled_elems(ix->n, ix->dim);
    VB_TRY(ix->base_hi.reserve(elems));
    if (ix->quant == VB200_QUANT_BF16) {
        VB_TRY(tc_pretile_bf16(ix->base_bf16.ptr, ix->n, ix->dim, ix->base_hi.ptr));
    } else {
        VB_TRY(ix->base_lo.reserve(elems));
        VB_TRY(tc_pretile_f32(ix->base_f32.ptr, ix->n, ix->dim, ix->base_hi.ptr, ix->base_lo.ptr));
    }
    ix->tiled_valid = true;
    ix->sample_stride = 0;
    return 0;
}

static int
bf_tile_queries(vb200_bf* ix, const float* q_dev, uint64_t nq) {
    const size_t q_elems = tc_tiled_elems(nq, ix->dim);
    VB_TRY(ix->q_hi.reserve(q_elems));
    if (ix->quant == VB200_QUANT_BF16) {
        return tc_pretile_bf16(ix->q_bf16.ptr, nq, ix->dim, ix->q_hi.ptr);
    }
    VB_TRY(ix->q_lo.reserve(q_elems));
    return tc_pretile_f32(q_dev, nq, ix->dim, ix->q_hi.ptr, ix->q_lo.ptr);
}

// Leaves the k best keys (payload = row) per query in ix->keys.
static int
bf_search_keys(vb200_bf* ix, const BfStaged& staged, uint64_t nq, uint32_t k) {
    const uint32_t dim = ix->dim;
    const uint64_t n = ix->n;
    uint32_t kcand = k + BF_SLACK;
    if (kcand > n) {
        kcand = static_cast<uint32_t>(n);
    }
    VB_CHECK_ARG(kcand <= 1024, "k = %u is too large (limit %u)", k, 1024 - BF_SLACK);
    const bool l2 = ix->metric == VB200_METRIC_L2;
    const bool bf16 = ix->quant == VB200_QUANT_BF16;
    const float *q_dev = staged.queries, *bias_all = staged.bias;
    // Large problems nominate candidates on the tensor cores; the exact re-scoring below is the
    // same either way.
    if (tensor_cores_enabled() && kcand <= tc_max_candidates(bf16 ? 1 : 3) && static_cast<double>(nq) * n * dim >= 2e10) {
        const uint32_t chunks = (dim + TC_KC - 1) / TC_KC;
        VB_TRY(bf_tile_base(ix));
        VB_TRY(bf_tile_queries(ix, q_dev, nq));
        TcOperand a{ix->q_hi.ptr, bf16 ? nullptr : ix->q_lo.ptr, nq, chunks, dim};
        VB_TRY(ix->cand.reserve(nq * kcand));
        VB_TRY(ix->row_bound.reserve(nq));
        // The base goes through the tensor cores in a few column ranges of growing size (a first one of about
        // a thousand rows, then sixteen times as many each time).  After each range the per-query candidate
        // lists are merged and the kcand-th score so far becomes the query's bound for the next range: no
        // column at or above it can be among the kcand best, so with rows in no particular order only about
        // 16 * kcand columns per query pass the bound in a range, and the kernel's per-row buffers hardly ever
        // need compacting.  Whatever the order of the rows, the result is the same set of candidates.
        const uint64_t n_tiles = (n + TC_BN - 1) / TC_BN;
        uint64_t len = n_tiles;
        if (n_tiles >= 1024) {
            len = 2 * kcand / TC_BN + 1 < 8 ? 8 : 2 * kcand / TC_BN + 1;
        }
        const uint32_t merge_cap = next_pow2(kcand + 256);
        const size_t merge_smem = merge_cap * sizeof(uint64_t) + 16;
        for (uint64_t tile0 = 0; tile0 < n_tiles; len *= 16) {
            uint64_t tile1 = tile0 + len;
            if (tile1 >= n_tiles || n_tiles - tile1 < len) {
                tile1 = n_tiles;   // no short last range
            }
            const uint64_t row0 = tile0 * TC_BN;
            const uint64_t rows = (tile1 * TC_BN < n ? tile1 * TC_BN : n) - row0;
            const size_t off = static_cast<size_t>(tile0) * chunks * TC_CHUNK_ELEMS;
            TcOperand b{ix->base_hi.ptr + off, bf16 ? nullptr : ix->base_lo.ptr + off, rows, chunks, dim};
            const bool first = tile0 == 0;
            uint32_t lists = 1;
            VB_TRY(tc_candidates(ix->tc, a, b, bf16 ? 1 : 3, l2 ? -2.0f : -1.0f, bias_all != nullptr ? bias_all + row0 : nullptr,
                                 kcand, static_cast<uint32_t>(row0), ix->tc_out, &lists, nullptr,
                                 first ? nullptr : ix->row_bound.ptr));
            VB_LAUNCH(bf_merge_kernel, static_cast<uint32_t>(nq), 256, merge_smem, ix->tc_out.ptr,
                      static_cast<uint64_t>(lists) * kcand, first ? static_cast<const uint64_t*>(nullptr) : ix->cand.ptr,
                      kcand, merge_cap, ix->cand.ptr, tile1 < n_tiles ? ix->row_bound.ptr : static_cast<float*>(nullptr));
            tile0 = tile1;
        }
        VB_TRY(ix->keys.reserve(nq * k));
        uint32_t n2 = next_pow2(kcand < 2 ? 2 : kcand);
        if (bf16) {
            VB_TRY(bf_rescore(ix->q_bf16.ptr, nq, dim, ix->base_bf16.ptr, ix->cand.ptr, kcand, n2, k, ix->metric, ix->keys.ptr));
        } else {
            VB_TRY(bf_rescore(q_dev, nq, dim, ix->base_f32.ptr, ix->cand.ptr, kcand, n2, k, ix->metric, ix->keys.ptr));
        }
        return 0;
    }
    const uint64_t col_chunk = n < BF_COL_CHUNK ? n : BF_COL_CHUNK;
    const uint32_t nchunks = static_cast<uint32_t>((n + col_chunk - 1) / col_chunk);
    uint64_t q_chunk = BF_SLAB_FLOATS / col_chunk;
    if (q_chunk < 1) {
        q_chunk = 1;
    }
    if (q_chunk > nq) {
        q_chunk = nq;
    }
    VB_TRY(ix->scores.reserve(q_chunk * col_chunk));
    const uint32_t keys_ld = nchunks * kcand;
    VB_TRY(ix->part.reserve(nq * keys_ld));
    for (uint64_t qb = 0; qb < nq; qb += q_chunk) {
        const uint64_t qn = nq - qb < q_chunk ? nq - qb : q_chunk;
        for (uint32_t c = 0; c < nchunks; ++c) {
            const uint64_t c0 = static_cast<uint64_t>(c) * col_chunk;
            const uint64_t cn = n - c0 < col_chunk ? n - c0 : col_chunk;
            const float* bias = bias_all != nullptr ? bias_all + c0 : nullptr;
            const float alpha = l2 ? -2.0f : -1.0f;
            if (bf16) {
                VB_TRY(dense_scores_bf16(ix->q_bf16.ptr + qb * dim, qn, ix->base_bf16.ptr + c0 * dim, cn,
                                         dim, alpha, bias, ix->scores.ptr, cn));
            } else {
                VB_TRY(dense_scores_f32(q_dev + qb * dim, qn, ix->base_f32.ptr + c0 * dim, cn, dim, alpha,
                                        bias, ix->scores.ptr, cn));
            }
            uint32_t kc = kcand < cn ? kcand : static_cast<uint32_t>(cn);
            if (kc < kcand) {  // short tail chunk: clear its slots first
                VB_CUDA(cudaMemset2DAsync(ix->part.ptr + qb * keys_ld + static_cast<uint64_t>(c) * kcand,
                                          keys_ld * sizeof(uint64_t), 0xFF, kcand * sizeof(uint64_t), qn,
                                          current_stream()));
            }
            VB_TRY(select_rows(ix->scores.ptr, qn, cn, cn, kc, static_cast<uint32_t>(c0),
                               ix->part.ptr + qb * keys_ld + static_cast<uint64_t>(c) * kcand, keys_ld));
        }
    }
    const uint64_t* cand = ix->part.ptr;
    if (nchunks > 1) {
        VB_TRY(ix->cand.reserve(nq * kcand));
        uint32_t cap = next_pow2(kcand + 256);
        size_t smem = cap * sizeof(uint64_t) + 16;
        VB_LAUNCH(bf_merge_kernel, static_cast<uint32_t>(nq), 256, smem, ix->part.ptr,
                  static_cast<uint64_t>(keys_ld), static_cast<const uint64_t*>(nullptr), kcand, cap, ix->cand.ptr,
                  static_cast<float*>(nullptr));
        cand = ix->cand.ptr;
    }
    VB_TRY(ix->keys.reserve(nq * k));
    uint32_t n2 = next_pow2(kcand < 2 ? 2 : kcand);
    if (bf16) {
        VB_TRY(bf_rescore(ix->q_bf16.ptr, nq, dim, ix->base_bf16.ptr, cand, kcand, n2, k, ix->metric, ix->keys.ptr));
    } else {
        VB_TRY(bf_rescore(q_dev, nq, dim, ix->base_f32.ptr, cand, kcand, n2, k, ix->metric, ix->keys.ptr));
    }
    return 0;
}

// Shared memory of a CTA that streams rows for qn queries, `keep` results each (no more than there are rows).
static uint32_t
bf_stream_cap(uint32_t keep) {
    return next_pow2(keep + RS_ROWS);
}

static size_t
bf_stream_smem(uint32_t dim, uint32_t cap, uint32_t qn) {
    return RS_STAGES * RS_STAGE + static_cast<size_t>(qn) * ((dim + 7) / 8 * 8) * sizeof(float) +
           static_cast<size_t>(qn) * (cap * sizeof(uint64_t) + 6 * sizeof(uint32_t));
}

// Exact distances of a few queries: one pass over the rows (bf_stream.cuh) straight to results in device or pinned memory.
// pick (optional, device): the queries' numbers among the staged ones, whose results go to the same numbers.
static int
bf_stream_queries(vb200_bf* ix, const BfStaged& staged, uint64_t nq, const uint32_t* pick, uint32_t k, int64_t* ids_dev, float* dists_dev) {
    const uint32_t dim = ix->dim;
    const bool l2 = ix->metric == VB200_METRIC_L2, bf16 = ix->quant == VB200_QUANT_BF16;
    BfStream p{};
    p.queries = bf16 ? static_cast<const void*>(ix->q_bf16.ptr) : staged.queries;
    p.pick = pick;
    p.nq = static_cast<uint32_t>(nq);
    p.dim = dim;
    p.base = bf16 ? reinterpret_cast<const unsigned char*>(ix->base_bf16.ptr) : reinterpret_cast<const unsigned char*>(ix->base_f32.ptr);
    p.n = ix->n;
    const uint32_t keep = static_cast<uint32_t>(std::min<uint64_t>(k, ix->n));
    p.k = keep;
    p.cap = bf_stream_cap(keep);
    p.masked = staged.masked ? staged.bias : nullptr;
    uint32_t qn = 1;
    while (qn < nq && qn < BF_STREAM_QUERIES) {
        qn *= 2;
    }
    while (qn > 1 && bf_stream_smem(dim, p.cap, qn) > 110 * 1024) {
        qn /= 2;
    }
    const size_t smem = bf_stream_smem(dim, p.cap, qn);
    VB_CHECK_ARG(smem <= 220 * 1024, "dim = %u is too large for the row scan", dim);
    const size_t row_bytes = static_cast<size_t>(dim) * (bf16 ? 2 : 4);
    const int unit = row_bytes % 16 == 0 ? 16 : (row_bytes % 4 == 0 ? 4 : 2);
    void (*kernel)(const BfStream) = nullptr;
#define VB_BF_UNIT(FMT, L2, QN)                                                                            \
    kernel = unit == 16 ? bf_stream_kernel<FMT, L2, QN, 16>                                                \
                        : (FMT == ROW_F32 || unit == 4 ? bf_stream_kernel<FMT, L2, QN, 4>                  \
                                                       : bf_stream_kernel<FMT, L2, QN, FMT == ROW_F32 ? 4 : 2>)
#define VB_BF_QN(FMT, L2)                          \
    switch (qn) {                                  \
        case 1: VB_BF_UNIT(FMT, L2, 1); break;     \
        case 2: VB_BF_UNIT(FMT, L2, 2); break;     \
        case 4: VB_BF_UNIT(FMT, L2, 4); break;     \
        default: VB_BF_UNIT(FMT, L2, 8); break;    \
    }
    if (bf16) {
        if (l2) {
            VB_BF_QN(ROW_BF16, true)
        } else {
            VB_BF_QN(ROW_BF16, false)
        }
    } else if (l2) {
        VB_BF_QN(ROW_F32, true)
    } else {
        VB_BF_QN(ROW_F32, false)
    }
#undef VB_BF_QN
#undef VB_BF_UNIT
    VB_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem));
    int per_sm = 0;
    VB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, RS_ROWS, smem));
    const uint64_t chunks = (ix->n + RS_ROWS - 1) / RS_ROWS;
    const uint32_t tiles = static_cast<uint32_t>((nq + qn - 1) / qn);
    // one wave of CTAs: with several tiles of queries each takes a larger share of the rows
    const uint64_t slots = static_cast<uint64_t>(sm_count()) * std::max(per_sm, 1);
    const uint32_t grid = static_cast<uint32_t>(std::min(chunks, std::max<uint64_t>(slots / tiles, 1)));
    VB_CHECK_ARG(nq * grid * keep < 0xFFFFFFFFull && tiles <= 65535, "query batch too large");
    VB_TRY(ix->part.reserve(nq * grid * keep));
    VB_TRY(ix->stream_bound.reserve(nq));
    VB_CUDA(cudaMemsetAsync(ix->stream_bound.ptr, 0xFF, nq * sizeof(uint32_t), current_stream()));
    p.part = ix->part.ptr;
    p.bound = ix->stream_bound.ptr;
    VB_LAUNCH(kernel, dim3(grid, tiles), RS_ROWS, smem, p);
    VB_LAUNCH(bf_pick_kernel<1024>, static_cast<uint32_t>(nq), 1024, 0, ix->part.ptr, grid * keep, keep, k, pick, ix->labels.ptr, ids_dev,
              dists_dev);
    return 0;
}

// Batches whose score matrix is worth writing: tensor-core scores in slices of queries,
// then a CTA per query that selects, re-scores and writes its results.  Leaves in ix->unsure the queries for which that
// may not have been enough.
// Slices of 512 MiB: with slices that stay in L2 (96 MiB) the launches are too short to fill the SMs, and the scores they
// save from a trip to HBM cost less than that (1000 queries over 100k x 128 rows: 8 slices 632 us, 4 517, 2 481, 1 431).
constexpr uint64_t BF_SLICE_SCORES = uint64_t{128} << 20;
constexpr uint64_t BF_UNSURE_SLICE = 4096;   // of those queries that are streamed at once (their partial results: k keys each per CTA)

static BfMargin
bf_margin(const vb200_bf* ix) {
    BfMargin margin{};
    margin.row_max = ix->row_max.ptr;
    margin.chain = static_cast<float>(ix->dim + 16) * 6.0e-8f;
    margin.matrix = ix->quant == VB200_QUANT_BF16 ? 2.0f * margin.chain : 4.0f * margin.chain + 3.0f / 262144.0f;
    margin.unsure = ix->unsure.ptr + 1;
    return margin;
}

// Batches over many rows: no score is written that a threshold rules out.
//   sample   one row in `stride`, and of every 32 of those the smallest score; of these minima the kcand-th smallest is a score
//            that kcand rows reach, so the rows with the kcand best scores are among those that do not pass it
//   collect  one pass over all rows appends what does not pass the query's threshold to its lists, about kcand * stride entries
//   rows     a CTA per query selects, re-scores and writes its results (bf_collected_kernel)
// 1000 queries over 100k x 128 fp32 rows, k 10: 13, 5, 75 and 47 us, where 121 wrote the scores and 174 selected from them.
struct BfSample {
    uint32_t stride = 0;       // 0: the rows are too few for a sample
    uint64_t groups = 0;       // of 32 rows in the sample
    double most = 0.0;         // rows that a query may collect
};
constexpr uint32_t BF_COLLECT_KEYS = 12288;          // of a query, at most (96 KiB of shared memory)
// Above this many products of one term the sample's share of them is more than the merges of bf_search_keys cost.  Calls of the two, ms:
//   10,000 queries  1M x 128 fp32 (3.8e12) k 10 5.7 / 7.8, k 100 6.7 / 10.8     200k x 768 fp32 (4.6e12) 8.6 / 9.8, 10.9 / 12.9
//                   6M x 256 bf16 (1.5e13) k 10 28.7 / 29.8, k 100 29.6 / 33.6  6M x 768 bf16 (4.8e13) k 100 89.2 / 87.2 (at the power limit)
//   and below: 3000 queries of 6M x 256 bf16 (4.6e12) 8.0 / 9.9, 300 (4.6e11) 1.1 / 2.0, 30 of 1M x 128 bf16 (3.8e9) 0.14 / 0.39.
constexpr double BF_COLLECT_PRODUCTS = 2e13;
constexpr uint32_t BF_COLLECT_DIMS = 16384;          // the query lies beside them
// List entries of the queries that go together, at most (2 GiB); where that is not to be had an eighth, and an eighth of that.
constexpr uint64_t BF_COLLECT_SLOTS = uint64_t{256} << 20, BF_COLLECT_LEAST = BF_COLLECT_SLOTS / 64;

// The sample takes a thirty-second of the rows, or the smallest larger power of two's share whose minima are four times kcand, so
// that the threshold is near the kcand-th best of the sample; at most an eighth, beyond which the scores are as well written.
// (A sixty-fourth lets twice as many rows pass: 6M x 768 rows, 10,000 queries, k 100: 1.8 ms for the sample and 72.9 for
// the pass, against 3.0 and 71.8.)
static BfSample
bf_sample(uint64_t n, uint32_t dim, uint32_t kcand) {
    BfSample s;
    if (dim > BF_COLLECT_DIMS) {
        return s;
    }
    for (uint32_t stride = 32; stride >= 8; stride /= 2) {
        const uint64_t minima = n / (32 * stride);
        // a row's chance to be below: of a minimum it is kcand / minima
        const double p = 1.0 - std::pow(1.0 - std::min(0.99, static_cast<double>(kcand) / static_cast<double>(minima)), 1.0 / 32.0);
        // what a query may collect: the threshold is the kcand-th of a sample, its rank in all rows known to 1 / sqrt(kcand);
        // six times that is room for all of a batch's queries (with 1.25 times the expected 31 of 10,000 did not fit)
        const double most = p * static_cast<double>(n) * (1.0 + 6.0 / std::sqrt(static_cast<double>(kcand))) + 256.0;
        if (minima >= 4ull * kcand && most <= BF_COLLECT_KEYS) {
            s.stride = stride;
            s.groups = minima;
            s.most = most;
            return s;
        }
    }
    return s;
}

// Row number `column` of a sample of `groups` times 32 of n rows.  The rows fall into as many stretches as the sample has rows, one
// is taken of each, somewhere in it, and neighbouring stretches go to different groups of 32: what the sample tells does not depend
// on the order of the rows.  (Whole tiles of 128 neighbours as a sample, with rows of a cluster stored together: the kcand-th
// minimum was that of a far cluster, every query collected more than it has room for, and the exact pass took the batch.)
__device__ __forceinline__ uint64_t
bf_sample_row(uint64_t column, uint64_t groups, uint64_t n) {
    const uint64_t total = groups * 32, s = (column & 31u) * groups + (column >> 5);
    const uint64_t first = s * n / total, width = (s + 1) * n / total - first;
    uint32_t h = static_cast<uint32_t>(s) * 0x9E3779B1u;   // (any fixed mixing of the bits: orders with a period are not in step with it)
    h = (h ^ (h >> 15)) * 0x85EBCA6Bu;
    h ^= h >> 13;
    return first + ((h * width) >> 32);
}

// The tiled terms and the score biases of the sample's rows, 16 bytes of a term per thread, rows before units.
__global__ void __launch_bounds__(256)
bf_sample_kernel(const uint4* __restrict__ hi, const uint4* __restrict__ lo, const float* __restrict__ bias, uint64_t n, uint64_t groups,
                 uint32_t chunks, uint4* __restrict__ out_hi, uint4* __restrict__ out_lo, float* __restrict__ out_bias) {
    const uint64_t e = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x;
    const uint64_t padded = (groups * 32 + TC_BN - 1) / TC_BN * TC_BN, column = e % padded;
    const uint32_t unit = static_cast<uint32_t>(e / padded);   // eight dimensions
    if (unit >= chunks * (TC_KC / 8)) {
        return;
    }
    const bool there = column < groups * 32;
    const uint64_t row = there ? bf_sample_row(column, groups, n) : 0;
    auto place = [&](uint64_t r) -> uint64_t {   // of the 16 bytes in the tiled layout (tc_pretile_kernel)
        return ((r / TC_BN * chunks + unit / 8) * 16 + r % TC_BN / 8) * 64 + unit % 8 * 8 + r % 8;
    };
    const uint4 none = make_uint4(0u, 0u, 0u, 0u);
    out_hi[place(column)] = there ? __ldg(hi + place(row)) : none;
    if (lo != nullptr) {
        out_lo[place(column)] = there ? __ldg(lo + place(row)) : none;
    }
    if (unit == 0 && there && bias != nullptr) {
        out_bias[column] = __ldg(bias + row);
    }
}

// Leaves the sample beside the tiled rows, where it stays until they change or a search wants another share of them.
static int
bf_take_sample(vb200_bf* ix, const BfSample& sample, const float* bias) {
    if (ix->sample_stride == sample.stride) {
        return 0;
    }
    ix->sample_stride = 0;
    const uint64_t rows = sample.groups * 32, elems = tc_tiled_elems(rows, ix->dim);
    const bool bf16 = ix->quant == VB200_QUANT_BF16;
    VB_TRY(ix->sample_hi.reserve(elems));
    VB_TRY(ix->sample_lo.reserve(bf16 ? 0 : elems));
    VB_TRY(ix->sample_bias.reserve(bias != nullptr ? rows : 0));
    const uint64_t blocks = (elems / 8 + 255) / 256;
    VB_CHECK_ARG(blocks <= 0x7fffffffu, "too many rows for a sample");
    VB_LAUNCH(bf_sample_kernel, static_cast<uint32_t>(blocks), 256, 0, reinterpret_cast<const uint4*>(ix->base_hi.ptr),
              bf16 ? static_cast<const uint4*>(nullptr) : reinterpret_cast<const uint4*>(ix->base_lo.ptr), bias, ix->n, sample.groups,
              (ix->dim + TC_KC - 1) / TC_KC, reinterpret_cast<uint4*>(ix->sample_hi.ptr), reinterpret_cast<uint4*>(ix->sample_lo.ptr),
              ix->sample_bias.ptr);
    ix->sample_stride = sample.stride;
    return 0;
}

static int
bf_search_collected(vb200_bf* ix, const BfStaged& staged, const BfSample& sample, uint64_t slots, uint64_t nq, uint32_t k, int64_t* ids_dev,
                    float* dists_dev) {
    const uint32_t dim = ix->dim;
    const bool l2 = ix->metric == VB200_METRIC_L2, bf16 = ix->quant == VB200_QUANT_BF16;
    const float* q_dev = staged.queries;
    const float alpha = l2 ? -2.0f : -1.0f;
    VB_TRY(bf_tile_base(ix));
    VB_TRY(bf_take_sample(ix, sample, staged.bias));
    VB_TRY(bf_tile_queries(ix, q_dev, nq));
    const uint32_t chunks = (dim + TC_KC - 1) / TC_KC, terms = bf16 ? 1 : 3;
    const uint32_t kcand = static_cast<uint32_t>(std::min<uint64_t>(k + BF_SLACK, ix->n));
    const uint64_t ld = (sample.groups + 3) / 4 * 4;   // (whole tiles; groups past the last are +inf)
    const uint32_t room = std::max<uint32_t>(512, std::min<uint32_t>(BF_COLLECT_KEYS, static_cast<uint32_t>(1.25 * sample.most) + 256));
    // whole row tiles whose lists fit
    TcCollect plan = tc_collect_plan(nq, ix->n, sample.most);
    uint64_t slice = slots / (static_cast<uint64_t>(plan.lists) * plan.cap + room) / TC_BM * TC_BM;
    slice = slice < TC_BM ? TC_BM : (slice > nq ? nq : slice);
    if (slice < nq) {
        const uint64_t parts = (nq + slice - 1) / slice;
        slice = ((nq + parts - 1) / parts + TC_BM - 1) / TC_BM * TC_BM;
        plan = tc_collect_plan(slice, ix->n, sample.most);
    }
    VB_TRY(ix->scores.reserve(slice * ld));
    VB_TRY(ix->row_bound.reserve(slice));
    VB_TRY(ix->tc_out.reserve(slice * plan.lists * plan.cap));
    VB_TRY(ix->list_count.reserve(slice * plan.lists));
    VB_TRY(ix->spill.reserve(slice * room));
    VB_TRY(ix->spilled.reserve(slice));
    VB_TRY(ix->unsure.reserve(nq + 2));
    VB_CUDA(cudaMemsetAsync(ix->unsure.ptr, 0, 2 * sizeof(uint32_t), current_stream()));
    int* const error_flag = reinterpret_cast<int*>(ix->unsure.ptr);
    const TcOperand b{ix->base_hi.ptr, bf16 ? nullptr : ix->base_lo.ptr, ix->n, chunks, dim};
    const TcOperand sampled{ix->sample_hi.ptr, bf16 ? nullptr : ix->sample_lo.ptr, sample.groups * 32, chunks, dim};
    const float* sampled_bias = staged.bias != nullptr ? ix->sample_bias.ptr : nullptr;
    BfCollected c{};
    c.keys = ix->tc_out.ptr;
    c.count = ix->list_count.ptr;
    c.thr = ix->row_bound.ptr;
    c.lists = plan.lists;
    c.cap = plan.cap;
    c.room = room;
    c.spill = ix->spill.ptr;
    c.spilled = ix->spilled.ptr;
    c.dim = dim;
    c.kcand = kcand;
    c.k = k;
    c.metric = ix->metric;
    c.labels = ix->labels.ptr;
    c.m = bf_margin(ix);
    const size_t smem = static_cast<size_t>(c.room) * sizeof(uint64_t) + (plan.lists + 2) * sizeof(uint32_t) + dim * sizeof(float);
    VB_CHECK_ARG(smem <= 180 * 1024, "dim = %u is too large for the exact re-scoring step", dim);
    for (uint64_t q0 = 0; q0 < nq; q0 += slice) {
        const uint64_t m = std::min(slice, nq - q0);
        const size_t off = static_cast<size_t>(q0 / TC_BM) * chunks * TC_CHUNK_ELEMS;
        const TcOperand a{ix->q_hi.ptr + off, bf16 ? nullptr : ix->q_lo.ptr + off, m, chunks, dim};
        VB_TRY(tc_minima(a, sampled, terms, alpha, sampled_bias, ix->scores.ptr, ld, error_flag));
        VB_LAUNCH(bf_threshold_kernel, static_cast<uint32_t>(m), BF_THRESHOLD_THREADS, 0, ix->scores.ptr, static_cast<uint32_t>(ld), kcand,
                  ix->row_bound.ptr, ix->spilled.ptr);
        VB_TRY(tc_collect(plan, a, b, terms, alpha, staged.bias, ix->row_bound.ptr, ix->tc_out.ptr, ix->list_count.ptr,
                          TcSpill{ix->spill.ptr, ix->spilled.ptr, room}, error_flag));
        c.queries = bf16 ? static_cast<const void*>(ix->q_bf16.ptr + q0 * dim) : q_dev + q0 * dim;
        c.base = bf16 ? static_cast<const void*>(ix->base_bf16.ptr) : ix->base_f32.ptr;
        c.ids = ids_dev + q0 * k;
        c.dists = dists_dev + q0 * k;
        c.m.q_base = static_cast<uint32_t>(q0);
        auto kernel = bf16 ? bf_collected_kernel<uint16_t, 512> : bf_collected_kernel<float, 512>;
        VB_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem));
        VB_LAUNCH(kernel, static_cast<uint32_t>(m), 512, smem, c);
    }
    return 0;
}

static int
bf_search_scores(vb200_bf* ix, const BfStaged& staged, uint64_t nq, uint32_t k, int64_t* ids_dev, float* dists_dev) {
    const uint32_t dim = ix->dim;
    const bool l2 = ix->metric == VB200_METRIC_L2, bf16 = ix->quant == VB200_QUANT_BF16;
    const float* q_dev = staged.queries;
    VB_TRY(bf_tile_base(ix));
    VB_TRY(bf_tile_queries(ix, q_dev, nq));
    const uint32_t chunks = (dim + TC_KC - 1) / TC_KC;
    const uint64_t ld = (ix->n + 127) / 128 * 128;
    uint64_t slice = BF_SLICE_SCORES / ld / TC_BM * TC_BM;   // whole row tiles
    slice = slice < TC_BM ? TC_BM : slice;
    VB_TRY(ix->scores.reserve(std::min(slice, nq) * ld));
    VB_TRY(ix->unsure.reserve(nq + 2));
    VB_CUDA(cudaMemsetAsync(ix->unsure.ptr, 0, 2 * sizeof(uint32_t), current_stream()));
    int* const error_flag = reinterpret_cast<int*>(ix->unsure.ptr);
    const TcOperand b{ix->base_hi.ptr, bf16 ? nullptr : ix->base_lo.ptr, ix->n, chunks, dim};
    const uint32_t kcand = static_cast<uint32_t>(std::min<uint64_t>(k + BF_SLACK, ix->n));
    const size_t smem = dim * sizeof(float);
    VB_CHECK_ARG(smem <= 180 * 1024, "dim = %u is too large for the exact re-scoring step", dim);
    BfMargin margin = bf_margin(ix);
    for (uint64_t q0 = 0; q0 < nq; q0 += slice) {
        const uint64_t m = std::min(slice, nq - q0);
        const size_t off = static_cast<size_t>(q0 / TC_BM) * chunks * TC_CHUNK_ELEMS;
        const TcOperand a{ix->q_hi.ptr + off, bf16 ? nullptr : ix->q_lo.ptr + off, m, chunks, dim};
        margin.q_base = static_cast<uint32_t>(q0);
        VB_TRY(tc_scores(ix->tc, a, b, bf16 ? 1 : 3, l2 ? -2.0f : -1.0f, staged.bias, ix->scores.ptr, ld, error_flag));
        if (bf16) {
            auto kernel = bf_rows_kernel<uint16_t, 512>;
            VB_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem));
            VB_LAUNCH(kernel, static_cast<uint32_t>(m), 512, smem, ix->scores.ptr, ld, static_cast<uint32_t>(ix->n),
                      ix->q_bf16.ptr + q0 * dim, dim, ix->base_bf16.ptr, kcand, k, ix->metric, ix->labels.ptr, ids_dev + q0 * k,
                      dists_dev + q0 * k, margin);
        } else {
            auto kernel = bf_rows_kernel<float, 512>;
            VB_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem));
            VB_LAUNCH(kernel, static_cast<uint32_t>(m), 512, smem, ix->scores.ptr, ld, static_cast<uint32_t>(ix->n), q_dev + q0 * dim, dim,
                      ix->base_f32.ptr, kcand, k, ix->metric, ix->labels.ptr, ids_dev + q0 * k, dists_dev + q0 * k, margin);
        }
    }
    return 0;
}

static int
bf_check_search(vb200_bf* ix, const float* queries, uint64_t nq, uint32_t k) {
    VB_CHECK_ARG(ix != nullptr, "null index");
    VB_CHECK_ARG(queries != nullptr || nq == 0, "query pointer is null");
    VB_CHECK_ARG(k >= 1, "k must be positive");
    return 0;
}

extern "C" int
vb200_bf_search(vb200_bf_t ix, const float* queries, uint64_t nq, uint32_t k, int64_t* ids,
                float* dists) {
    return vb200_bf_search_filtered(ix, queries, nq, k, nullptr, ids, dists);
}

extern "C" int
vb200_bf_search_filtered(vb200_bf_t ix, const float* queries, uint64_t nq, uint32_t k, const vb200_filter* filter,
                         int64_t* ids, float* dists) {
    VB_TRY(bf_check_search(ix, queries, nq, k));
    if (nq == 0) {
        return 0;
    }
    VB_CHECK_ARG(ids != nullptr && dists != nullptr, "null output pointer");
    std::lock_guard<std::mutex> lock(ix->mu);
    const uint64_t total = nq * k;
    if (ix->n == 0) {
        std::vector<int64_t> hi(total, -1);
        std::vector<float> hd(total, INFINITY);
        VB_CUDA(cudaMemcpy(ids, hi.data(), total * sizeof(int64_t), cudaMemcpyDefault));
        VB_CUDA(cudaMemcpy(dists, hd.data(), total * sizeof(float), cudaMemcpyDefault));
        return 0;
    }
    // results go straight to device buffers, or to pinned memory when they are small; else through buffers here
    const bool host_ids = !is_device_pointer(ids), host_d = !is_device_pointer(dists);
    const bool pin_out = (host_ids || host_d) && total * 12 <= BF_PINNED_BYTES;
    if (pin_out) {
        VB_TRY(ix->pinned.reserve(total * 12));
    } else {
        if (host_ids) {
            VB_TRY(ix->out_ids.reserve(total));
        }
        if (host_d) {
            VB_TRY(ix->out_dists.reserve(total));
        }
    }
    int64_t* pin_ids = static_cast<int64_t*>(ix->pinned.ptr);
    float* pin_dists = pin_out ? reinterpret_cast<float*>(pin_ids + total) : nullptr;
    int64_t* ids_dev = !host_ids ? ids : (pin_out ? pin_ids : ix->out_ids.ptr);
    float* dists_dev = !host_d ? dists : (pin_out ? pin_dists : ix->out_dists.ptr);
    const bool k_fits = std::min<uint64_t>(k + BF_SLACK, ix->n) <= 1024;
    // (rows too long for a stream's shared memory, above 40,000 dimensions, are left to the slab of scores)
    const bool streams = k_fits && bf_stream_smem(ix->dim, bf_stream_cap(static_cast<uint32_t>(std::min<uint64_t>(k, ix->n))), 1) <= 220 * 1024;
    const bool few = nq <= BF_STREAM_QUERIES && streams;
    const bool batch = tensor_cores_enabled() && streams && !few;
    bool scores = batch && static_cast<double>(nq) * ix->n <= BF_MATRIX_SCORES, collected = false;
    BfStaged staged;
    bool keyed = false;
    ix->filter = filter;
    int rc = bf_stage(ix, queries, nq, &staged);
    // Up to eight queries share one pass over the rows; more go to the tensor cores, which keep what passes a threshold from a
    // sample of the rows; where the sample would be a large part of them, or rows are filtered out, through a score matrix
    // while that is cheaper than selecting as the scores appear (measured: up to about 4e8 scores), see
    // bf_search_keys for the rest.
    if (rc == 0 && few) {
        rc = bf_stream_queries(ix, staged, nq, nullptr, k, ids_dev, dists_dev);
    } else if (rc == 0 && batch) {
        const BfSample sample = staged.masked ? BfSample{} : bf_sample(ix->n, ix->dim, static_cast<uint32_t>(std::min<uint64_t>(k + BF_SLACK, ix->n)));
        const double products = static_cast<double>(nq) * ix->n * ix->dim * (ix->quant == VB200_QUANT_BF16 ? 1 : 3);
        collected = sample.stride != 0 && products <= BF_COLLECT_PRODUCTS;
        auto out_of_memory = [&]() -> bool {   // then what the attempt has taken is given back
            if (rc != VB200_NO_ENOUGH_MEMORY) {
                return false;
            }
            (void)cudaStreamSynchronize(current_stream());
            if (!ix->tiled_valid) {
                ix->base_hi.release();
                ix->base_lo.release();
            }
            ix->scores.release();
            ix->tc_out.release();
            ix->spill.release();
            rc = 0;
            return true;
        };
        for (uint64_t slots = BF_COLLECT_SLOTS; collected; slots /= 8) {
            rc = bf_search_collected(ix, staged, sample, slots, nq, k, ids_dev, dists_dev);
            if (!out_of_memory()) {
                break;
            }
            // (the tiled copy of the rows may be what did not fit)
            collected = ix->tiled_valid && slots > BF_COLLECT_LEAST;
            scores = scores && ix->tiled_valid;
        }
        if (rc == 0 && scores && !collected) {
            rc = bf_search_scores(ix, staged, nq, k, ids_dev, dists_dev);
            scores = !out_of_memory();   // (the slab of scores needs no tiled copy)
        }
    }
    if (rc == 0 && !few && !scores && !collected) {
        rc = bf_search_keys(ix, staged, nq, k);
        keyed = true;
    }
    ix->filter = nullptr;
    VB_TRY(rc);
    if (keyed) {
        VB_LAUNCH(bf_results_kernel, static_cast<uint32_t>((total + 255) / 256), 256, 0, ix->keys.ptr, total, ix->labels.ptr, ids_dev,
                  dists_dev, nullptr);
    }
    auto results_to_host = [&]() -> int {
        if (!pin_out) {
            if (host_ids) {
                VB_CUDA(cudaMemcpyAsync(ids, ids_dev, total * sizeof(int64_t), cudaMemcpyDeviceToHost, current_stream()));
            }
            if (host_d) {
                VB_CUDA(cudaMemcpyAsync(dists, dists_dev, total * sizeof(float), cudaMemcpyDeviceToHost, current_stream()));
            }
        }
        return 0;
    };
    VB_TRY(results_to_host());
    uint32_t report[2] = {0, 0};   // of the batch's kernels: error flag, unsure queries
    if (scores || collected) {
        VB_CUDA(cudaMemcpyAsync(report, ix->unsure.ptr, sizeof(report), cudaMemcpyDeviceToHost, current_stream()));
    }
    VB_TRY(sync_stream());
    if ((report[0] & 1) != 0) {
        VB_FAIL(VB200_INTERNAL_ERROR, "tensor-core kernel gave up on a bounded wait");
    }
    if (report[1] > 0) {
        for (uint64_t u0 = 0; u0 < report[1]; u0 += BF_UNSURE_SLICE) {
            VB_TRY(bf_stream_queries(ix, staged, std::min<uint64_t>(BF_UNSURE_SLICE, report[1] - u0), ix->unsure.ptr + 2 + u0, k, ids_dev,
                                     dists_dev));
        }
        VB_TRY(results_to_host());
        VB_TRY(sync_stream());
    }
    if (pin_out) {
        if (host_ids) {
            std::memcpy(ids, ids_dev, total * sizeof(int64_t));
        }
        if (host_d) {
            std::memcpy(dists, dists_dev, total * sizeof(float));
        }
    }
    return 0;
}

extern "C" int
vb200_bf_search_partial(vb200_bf_t ix, const float* queries, uint64_t nq, uint32_t k,
                        uint64_t* keys_dev, int64_t* labels_dev) {
    VB_TRY(bf_check_search(ix, queries, nq, k));
    if (nq == 0) {
        return 0;
    }
    VB_CHECK_ARG(keys_dev != nullptr && labels_dev != nullptr, "null output pointer");
    VB_CHECK_ARG(is_device_pointer(keys_dev) && is_device_pointer(labels_dev),
                 "partial results are written to device memory");
    std::lock_guard<std::mutex> lock(ix->mu);
    const uint64_t total = nq * k;
    if (ix->n == 0) {
        VB_CUDA(cudaMemsetAsync(keys_dev, 0xFF, total * sizeof(uint64_t), current_stream()));
        VB_CUDA(cudaMemsetAsync(labels_dev, 0xFF, total * sizeof(int64_t), current_stream()));
        return sync_stream();
    }
    BfStaged staged;
    VB_TRY(bf_stage(ix, queries, nq, &staged));
    VB_TRY(bf_search_keys(ix, staged, nq, k));
    VB_LAUNCH(bf_results_kernel, static_cast<uint32_t>((total + 255) / 256), 256, 0, ix->keys.ptr, total,
              ix->labels.ptr, labels_dev, nullptr, keys_dev);
    return sync_stream();
}

extern "C" int
vb200_bf_search_sharded(vb200_bf_t ix, vb200_comm_t comm, const float* queries, uint64_t nq, uint32_t k,
                        int64_t* ids, float* dists) {
    VB_CHECK_ARG(comm != nullptr, "null communicator");
    if (comm->world == 1) {
        return vb200_bf_search(ix, queries, nq, k, ids, dists);
    }
    VB_TRY(bf_check_search(ix, queries, nq, k));
    if (nq == 0) {
        return 0;
    }
    VB_CHECK_ARG(ids != nullptr && dists != nullptr, "null output pointer");
    std::lock_guard<std::mutex> lock(ix->mu);
    cudaStream_t st = current_stream();
    const uint64_t total = nq * k;
    const uint32_t world = static_cast<uint32_t>(comm->world);
    VB_TRY(ix->sh_local.reserve(2 * total));
    VB_TRY(ix->sh_all.reserve(static_cast<size_t>(world) * 2 * total));
    if (ix->n == 0) {
        VB_CUDA(cudaMemsetAsync(ix->sh_local.ptr, 0xFF, 2 * total * sizeof(uint64_t), st));
    } else {
        BfStaged staged;
        VB_TRY(bf_stage(ix, queries, nq, &staged));
        VB_TRY(bf_search_keys(ix, staged, nq, k));
        VB_LAUNCH(bf_results_kernel, static_cast<uint32_t>((total + 255) / 256), 256, 0, ix->keys.ptr, total,
                  ix->labels.ptr, reinterpret_cast<int64_t*>(ix->sh_local.ptr + total), nullptr, ix->sh_local.ptr);
    }
    VB_TRY(comm_all_gather(comm, ix->sh_local.ptr, ix->sh_all.ptr, 2 * total * sizeof(uint64_t), st));
    VB_TRY(merge_partials_device(ix->sh_all.ptr, reinterpret_cast<const int64_t*>(ix->sh_all.ptr + total), world,
                                 2 * total, nq, k, ids, dists));
    return sync_stream();
}
