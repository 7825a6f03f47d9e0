// k-means Lloyd iterations for IVF partition training: exact assignment through the fixed-order
// dense kernel with a fused argmin epilogue, and the centroid update.
#include "kmeans.cuh"

#include <algorithm>
#include <random>
#include <vector>

#include <cmath>
#include <cstdlib>

#include <cub/device/device_radix_sort.cuh>

#include "dense.cuh"
#include "kpp.cuh"

namespace vb200 {

// err += sum_i double(best_i + |x_i|^2) (src/impl/cluster/kmeans_cluster.cpp:281-296).
__global__ void __launch_bounds__(256)
kmeans_error_kernel(const float* __restrict__ x_sq, uint64_t n, const float* __restrict__ best, double* __restrict__ err) {
    __shared__ double partial[8];
    double v = 0.0;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x; i < n; i += static_cast<uint64_t>(gridDim.x) * 256) {
        v += static_cast<double>(__fadd_rn(best[i], x_sq[i]));
    }
    for (int off = 16; off > 0; off >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, off);
    }
    if ((threadIdx.x & 31) == 0) {
        partial[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < 8; ++w) {
            s += partial[w];
        }
        atomicAdd(err, s);
    }
}

static std::atomic<int> g_tc_enabled{-1};

bool
tensor_cores_enabled() {
    int v = g_tc_enabled.load();
    if (v < 0) {
        const char* e = getenv("VB200_DISABLE_TC");
        v = (e != nullptr && e[0] != 0 && e[0] != '0') ? 0 : 1;
        g_tc_enabled.store(v);
    }
    return v == 1;
}

// The pick among each row's candidate centroids: the one the reference's arithmetic prefers, score = fma(-2, <c, x>,
// |c|^2) with the inner product as one ascending FMA chain, lowest index on ties
// (src/impl/cluster/kmeans_cluster.cpp:262-284).  Candidates whose nominating score lies further than the row's margin
// behind the best one cannot be it; when a single one is left -- nearly always -- it needs no exact score, unless the
// caller wants the score itself (best_out).  The rows with more go to a list, whose rows take four lanes each: scored
// on the spot, two such rows of a warp kept the other thirty lanes waiting for their chains (390 us a pass over 1M rows).
__device__ __forceinline__ float
kmeans_exact_score(const float* __restrict__ c, const float* __restrict__ x, uint32_t dim, float c_sq, bool vec) {
    float ip = 0.f;
    if (vec) {
        // (operands fetched 64 bytes ahead of the chain)
        for (uint32_t d = 0; d < dim; d += 16) {
            float4 cv[4], xv[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                if (d + 4 * u < dim) {
                    cv[u] = __ldg(reinterpret_cast<const float4*>(c + d) + u);
                    xv[u] = __ldg(reinterpret_cast<const float4*>(x + d) + u);
                }
            }
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                if (d + 4 * u < dim) {
                    ip = fmaf(cv[u].x, xv[u].x, ip);
                    ip = fmaf(cv[u].y, xv[u].y, ip);
                    ip = fmaf(cv[u].z, xv[u].z, ip);
                    ip = fmaf(cv[u].w, xv[u].w, ip);
                }
            }
        }
    } else {
        for (uint32_t d = 0; d < dim; ++d) {
            ip = fmaf(__ldg(c + d), __ldg(x + d), ip);
        }
    }
    return fmaf(-2.0f, ip, c_sq);
}

constexpr uint32_t PICK_LANES = 4;

__global__ void __launch_bounds__(256)
kmeans_single_kernel(uint64_t n, const uint64_t* __restrict__ cand, uint32_t per_row, const float* __restrict__ row_margin,
                     int32_t* __restrict__ labels, uint32_t* __restrict__ close) {
    const uint64_t i = (static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x) / PICK_LANES;
    const uint32_t sub = threadIdx.x % PICK_LANES;
    const uint64_t* ci = cand + i * per_row;
    uint64_t least = KEY_INF, next = KEY_INF;   // the two smallest keys of this lane, then of the row
    if (i < n) {
        for (uint32_t j = sub; j < per_row; j += PICK_LANES) {
            const uint64_t key = __ldg(ci + j);
            next = key < least ? least : (key < next ? key : next);
            least = key < least ? key : least;
        }
    }
#pragma unroll
    for (uint32_t off = PICK_LANES >> 1; off > 0; off >>= 1) {
        const uint64_t a = __shfl_xor_sync(0xffffffffu, least, off), b = __shfl_xor_sync(0xffffffffu, next, off);
        next = a < least ? (least < b ? least : b) : (a < next ? a : next);
        least = a < least ? a : least;
    }
    if (i >= n || sub != 0) {
        return;
    }
    if (least == KEY_INF) {
        labels[i] = 0;
        return;
    }
    labels[i] = static_cast<int32_t>(static_cast<uint32_t>(least));
    if (next != KEY_INF &&
        ordered_to_float(static_cast<uint32_t>(next >> 32)) <= ordered_to_float(static_cast<uint32_t>(least >> 32)) + __ldg(row_margin + i)) {
        close[1 + atomicAdd(close, 1u)] = static_cast<uint32_t>(i);
    }
}

// Exact scores of the candidates of the rows in close[1 .. close[0]] (null: of all n rows), four lanes per row.
__global__ void __launch_bounds__(256)
kmeans_pick_kernel(const float* __restrict__ x, uint64_t n, uint32_t dim, const float* __restrict__ centroids,
                   const float* __restrict__ c_sq, const uint64_t* __restrict__ cand, uint32_t per_row,
                   const float* __restrict__ row_margin, const uint32_t* __restrict__ close, int32_t* __restrict__ labels,
                   float* __restrict__ best_out) {
    const uint64_t count = close != nullptr ? close[0] : n;
    const uint32_t sub = threadIdx.x % PICK_LANES;
    const bool vec = (dim & 3u) == 0 && ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(centroids)) & 15u) == 0;
    const uint64_t step = static_cast<uint64_t>(gridDim.x) * 256 / PICK_LANES;
    for (uint64_t e0 = static_cast<uint64_t>(blockIdx.x) * 256 / PICK_LANES; e0 < count; e0 += step) {
        const uint64_t e = e0 + threadIdx.x / PICK_LANES;
        const bool live = e < count;
        const uint64_t i = !live ? 0 : (close != nullptr ? close[1 + e] : e);
        const uint64_t* ci = cand + i * per_row;
        uint64_t least = KEY_INF;
        if (live) {
            for (uint32_t j = sub; j < per_row; j += PICK_LANES) {
                const uint64_t key = __ldg(ci + j);
                least = key < least ? key : least;
            }
        }
#pragma unroll
        for (uint32_t off = PICK_LANES >> 1; off > 0; off >>= 1) {
            const uint64_t other = __shfl_xor_sync(0xffffffffu, least, off);
            least = other < least ? other : least;
        }
        float best = INFINITY;
        uint32_t best_col = 0x7fffffffu;
        if (live && least != KEY_INF) {
            const float limit = ordered_to_float(static_cast<uint32_t>(least >> 32)) + __ldg(row_margin + i);
            // the row's candidates within the limit, dealt to its lanes in turn
            uint32_t turn = 0;
            for (uint32_t j = 0; j < per_row; ++j) {
                const uint64_t key = __ldg(ci + j);
                if (key == KEY_INF || ordered_to_float(static_cast<uint32_t>(key >> 32)) > limit) {
                    continue;
                }
                if (turn++ % PICK_LANES != sub) {
                    continue;
                }
                const uint32_t col = static_cast<uint32_t>(key);
                const float score = kmeans_exact_score(centroids + static_cast<uint64_t>(col) * dim, x + i * dim, dim, __ldg(c_sq + col), vec);
                if (score < best || (score == best && col < best_col)) {
                    best = score;
                    best_col = col;
                }
            }
        }
#pragma unroll
        for (uint32_t off = PICK_LANES >> 1; off > 0; off >>= 1) {
            float ob = __shfl_xor_sync(0xffffffffu, best, off);
            uint32_t oc = __shfl_xor_sync(0xffffffffu, best_col, off);
            if (ob < best || (ob == best && oc < best_col)) {
                best = ob;
                best_col = oc;
            }
        }
        if (live && sub == 0) {
            labels[i] = best_col == 0x7fffffffu ? 0 : static_cast<int32_t>(best_col);
            if (best_out != nullptr) {
                best_out[i] = best;
            }
        }
    }
}

// shift[d] = mean of the centroids' component d.  A CTA per 32 components.
__global__ void __launch_bounds__(1024)
kmeans_shift_kernel(const float* __restrict__ c, uint32_t k, uint32_t dim, float* __restrict__ shift) {
    __shared__ float part[32][33];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d = blockIdx.x * 32 + lane;
    float s = 0.f;
    for (uint32_t j = warp; d < dim && j < k; j += 32) {
        s += c[static_cast<uint64_t>(j) * dim + d];
    }
    part[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && d < dim) {
        for (int w = 1; w < 32; ++w) {
            s += part[w][lane];
        }
        shift[d] = s / static_cast<float>(k);
    }
}

// Norms of the rows as they are and shifted (rounded up; null: not wanted), the largest |element| of the shifted rows
// and the largest norms.  A warp per row.  shifted (optional): the shifted rows.
__global__ void __launch_bounds__(256)
kmeans_norms_kernel(const float* __restrict__ x, uint64_t n, uint32_t dim, const float* __restrict__ shift, float* __restrict__ norm,
                    float* __restrict__ shifted_norm, float* __restrict__ shifted, float* __restrict__ max_element,
                    float* __restrict__ max_norms) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warps = static_cast<uint64_t>(gridDim.x) * 8;
    float top = 0.f, top_s = 0.f, top_n = 0.f;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * 8 + (threadIdx.x >> 5); i < n; i += warps) {
        float a = 0.f, b = 0.f;
        for (uint32_t d = lane; d < dim; d += 32) {
            const float v = x[i * dim + d], w = v - shift[d];
            a = fmaf(v, v, a);
            b = fmaf(w, w, b);
            top = fmaxf(top, fabsf(w));
            if (w != w) {
                top = INFINITY;
            }
            if (shifted != nullptr) {
                shifted[i * dim + d] = w;
            }
        }
        for (int off = 16; off > 0; off >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, off);
            b += __shfl_xor_sync(0xffffffffu, b, off);
        }
        a = sqrtf(a) * 1.0001f;
        b = sqrtf(b) * 1.0001f;
        if (lane == 0 && norm != nullptr) {
            norm[i] = a;
            shifted_norm[i] = b;
        }
        top_n = fmaxf(top_n, a);
        top_s = fmaxf(top_s, b);
    }
    for (int off = 16; off > 0; off >>= 1) {
        top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, off));
    }
    if (lane == 0) {   // non-negative floats order like their bit patterns
        atomicMax(reinterpret_cast<int*>(max_element), __float_as_int(top));
        if (max_norms != nullptr) {
            atomicMax(reinterpret_cast<int*>(max_norms), __float_as_int(top_s));
            atomicMax(reinterpret_cast<int*>(max_norms) + 1, __float_as_int(top_n));
        }
    }
}

// margin[i] = by_shifted * max|c - shift| * |x_i - shift| + by_plain * max|c| * |x_i| + by_square * max|c - shift|^2, and with `prev`
// bound[i] = the row's score against its previous centroid, |c'|^2 - 2 <c', x'> over shifted vectors (+inf when it has none), both
// in units of the products (times `unit`); to the margin, in those units, floor_each (max|c - shift| + |x_i - shift|) + floor.  Eight
// lanes per row.  Centroids that do not fit the fp16 scale (limit) leave no column out: the margin becomes infinite.
__global__ void __launch_bounds__(256)
kmeans_row_prep_kernel(const float* __restrict__ x, uint64_t n, uint32_t dim, const float* __restrict__ shift,
                       const float* __restrict__ c_shifted, const float* __restrict__ cs_sq, uint32_t k, const int32_t* __restrict__ prev,
                       const float* __restrict__ x_norm, const float* __restrict__ xs_norm, const float* __restrict__ extremes,
                       float by_shifted, float by_plain, float by_square, float floor_each, float floor, float limit, float unit,
                       float* __restrict__ margin, float* __restrict__ bound) {
    const uint64_t i = (static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x) >> 3;
    const uint32_t sub = threadIdx.x & 7u;
    if (i < n && sub == 0) {
        const float m = by_shifted * extremes[1] * xs_norm[i] + by_plain * extremes[2] * x_norm[i] + by_square * extremes[1] * extremes[1];
        margin[i] = extremes[0] <= limit ? m * unit + (floor_each * (extremes[1] + xs_norm[i]) + floor) : INFINITY;
    }
    if (prev == nullptr) {
        return;
    }
    int32_t l = -1;
    float ip = 0.f;
    if (i < n) {
        l = prev[i];
        if (l >= 0 && static_cast<uint32_t>(l) < k) {
            const float* xi = x + i * dim;
            const float* c = c_shifted + static_cast<uint64_t>(l) * dim;
            if ((dim & 3u) == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0) {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
                for (uint32_t d = sub * 4; d < dim; d += 32) {
                    const float4 xv = __ldg(reinterpret_cast<const float4*>(xi + d)), cv = __ldg(reinterpret_cast<const float4*>(c + d)),
                                 sv = __ldg(reinterpret_cast<const float4*>(shift + d));
                    acc[0] = fmaf(xv.x - sv.x, cv.x, acc[0]);
                    acc[1] = fmaf(xv.y - sv.y, cv.y, acc[1]);
                    acc[2] = fmaf(xv.z - sv.z, cv.z, acc[2]);
                    acc[3] = fmaf(xv.w - sv.w, cv.w, acc[3]);
                }
                ip = (acc[0] + acc[1]) + (acc[2] + acc[3]);
            } else {
                for (uint32_t d = sub; d < dim; d += 8) {
                    ip = fmaf(__ldg(xi + d) - __ldg(shift + d), __ldg(c + d), ip);
                }
            }
        }
    }
    for (int off = 4; off > 0; off >>= 1) {
        ip += __shfl_xor_sync(0xffffffffu, ip, off);
    }
    if (i < n && sub == 0) {
        bound[i] = l >= 0 && static_cast<uint32_t>(l) < k ? fmaf(-2.0f, ip, __ldg(cs_sq + l)) * unit : INFINITY;
    }
}

// The best centroid of the rows in `rows` over all centroids, exactly, as keys: grid.x = a few rows, grid.y = shares of
// the centroids, which stream through shared memory (as a matrix product over 128-row tiles a few rows took one CTA
// 560 us, as a CTA per row with the centroids read by a thread each 75 us).
template <int UNIT>
__global__ void __launch_bounds__(RS_ROWS)
kmeans_few_rows_kernel(const float* __restrict__ x, uint32_t dim, const float* __restrict__ centroids, const float* __restrict__ c_sq,
                       uint32_t k, const uint32_t* __restrict__ rows, unsigned long long* __restrict__ keys) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* xs = reinterpret_cast<float*>(smem + RS_STAGES * RS_STAGE);
    const uint64_t i = rows[blockIdx.x];
    const uint32_t qpad = (dim + 3) / 4 * 4;
    for (uint32_t d = threadIdx.x; d < qpad; d += RS_ROWS) {
        xs[d] = d < dim ? x[i * dim + d] : 0.f;
    }
    uint64_t mine = KEY_INF;
    RowAcc<ROW_F32, false, 1> acc;
    row_stream<UNIT>(reinterpret_cast<const unsigned char*>(centroids), static_cast<uint64_t>(dim) * 4, dim * 4, dim, k, blockIdx.y,
                     gridDim.y, smem, xs, qpad, acc, [&](uint64_t j, bool valid) {
                         if (valid) {
                             const uint64_t key = make_key(fmaf(-2.0f, acc.acc[0], __ldg(c_sq + j)), static_cast<uint32_t>(j));
                             mine = key < mine ? key : mine;
                         }
                     });
    for (int off = 16; off > 0; off >>= 1) {
        const uint64_t other = __shfl_xor_sync(0xffffffffu, mine, off);
        mine = other < mine ? other : mine;
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(keys + blockIdx.x, static_cast<unsigned long long>(mine));
    }
}

__global__ void
kmeans_keys_to_labels_kernel(const unsigned long long* __restrict__ keys, uint32_t count, const uint32_t* __restrict__ rows,
                             int32_t* __restrict__ labels, float* __restrict__ best_out) {
    const uint32_t e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < count) {
        labels[rows[e]] = static_cast<int32_t>(static_cast<uint32_t>(keys[e]));
        if (best_out != nullptr) {
            best_out[rows[e]] = ordered_to_float(static_cast<uint32_t>(keys[e] >> 32));
        }
    }
}

// rows[c] = i for every flagged row i (order irrelevant), *count = how many.
__global__ void
kmeans_collect_flagged_kernel(const uint32_t* __restrict__ flags, uint64_t n, uint32_t* __restrict__ rows,
                              uint32_t* __restrict__ count) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n && flags[i] != 0) {
        rows[atomicAdd(count, 1u)] = static_cast<uint32_t>(i);
    }
}

__global__ void
kmeans_gather_rows_kernel(const float* __restrict__ x, uint32_t dim, const uint32_t* __restrict__ rows, uint64_t count,
                          float* __restrict__ out) {
    const uint64_t e = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (e < count * dim) {
        out[e] = x[static_cast<uint64_t>(rows[e / dim]) * dim + e % dim];
    }
}

__global__ void
kmeans_scatter_labels_kernel(const uint32_t* __restrict__ rows, uint64_t count, const int32_t* __restrict__ lab,
                             const float* __restrict__ best, int32_t* __restrict__ labels, float* __restrict__ best_out) {
    const uint64_t c = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (c < count) {
        labels[rows[c]] = lab[c];
        if (best_out != nullptr) {
            best_out[rows[c]] = best[c];
        }
    }
}

constexpr uint32_t KMEANS_TC_CANDIDATES = 4;
constexpr uint64_t KMEANS_TC_SLICE = uint64_t{1} << 22;  // rows tiled at once
constexpr uint32_t KMEANS_FEW_ROWS = 4096;               // undecided rows that CTAs of their own decide

// Assignment through the tensor cores: candidates nominated by approximate scores, winner by the exact rule above.
//
// The scores are |c'|^2 - 2 <c', x'> over vectors minus a common shift (the centroids' mean: it changes no comparison
// of a row and takes the data's offset out of the errors), with x' and c' rounded to one fp16 term each, scaled so that
// the largest element is near 2^top: an error of at most 2 (2 * 2^-11 + 2^-22) |x'| |c'| per score, and of the sums, which hold |c'|^2
// among their products, (dim + 16) 2^-23 |c'|^2.  Scaled elements below 2^-14 round absolutely, by 2^-25, which is 2^-25 sqrt(dim) (|x'| + |c'|) of a
// scaled product, and the last of the bias's three terms by 2^-25 * 2^-7: next to nothing for rows of one size, and everything for the rows of
// ordinary size beside one that is 1e8 times as large, whose scaled squares vanish.  A column further
// than twice that (plus the rounding of the reference's own chain) behind a row's best is not its winner; the columns
// within are scored exactly.  A third of the MMAs that split bf16 terms take; those (2^-16 of the plain norms) remain for data
// whose shifted rows still crowd within the fp16 margin -- when more than a sixteenth of the rows came out undecided.
static int
kmeans_assign_tc(KMeansWorkspace& ws, const float* x_dev, uint64_t n, uint32_t dim,
                 const float* centroids_dev, uint32_t k, int32_t* labels_dev, float* best_dev,
                 const int32_t* prev_labels_dev) {
    const size_t c_elems = tc_tiled_elems(k, dim + TC_BIAS_DIMS);
    // Elements are scaled to below 2^top: the sum of their squares, whose half is a column's bias, stays below 2^30.
    int top_exponent = 14;
    while (top_exponent > 1 && std::ldexp(static_cast<double>(dim), 2 * top_exponent) > std::ldexp(1.0, 30)) {
        --top_exponent;
    }
    cudaStream_t st = current_stream();
    const uint32_t norm_blocks = 16u * static_cast<uint32_t>(sm_count());
    VB_TRY(ws.c_hi.reserve(c_elems));
    VB_TRY(ws.shift.reserve((dim + 3) / 4 * 4));
    VB_TRY(ws.c_shifted.reserve(static_cast<size_t>(k) * dim));
    VB_TRY(ws.cs_sq.reserve(k));
    VB_TRY(ws.extremes.reserve(3));
    const uint32_t m = k < KMEANS_TC_CANDIDATES ? k : KMEANS_TC_CANDIDATES;
    for (uint64_t r0 = 0; r0 < n; r0 += KMEANS_TC_SLICE) {
        const uint64_t rows = n - r0 < KMEANS_TC_SLICE ? n - r0 : KMEANS_TC_SLICE;
        const bool whole = rows == n;
        const bool cached = whole && ws.tiled_rows == x_dev && ws.tiled_n == n && ws.tiled_dim == dim;
        if (!cached) {
            const size_t x_elems = tc_tiled_elems(rows, dim + TC_BIAS_DIMS);
            VB_TRY(ws.x_hi.reserve(x_elems));
            VB_TRY(ws.x_norm.reserve(rows));
            VB_TRY(ws.xs_norm.reserve(rows));
            VB_CUDA(cudaMemsetAsync(ws.extremes.ptr, 0, 3 * sizeof(float), st));
            VB_LAUNCH(kmeans_shift_kernel, (dim + 31) / 32, 1024, 0, centroids_dev, k, dim, ws.shift.ptr);
            VB_LAUNCH(kmeans_norms_kernel, norm_blocks, 256, 0, x_dev + r0 * dim, rows, dim, ws.shift.ptr, ws.x_norm.ptr, ws.xs_norm.ptr,
                      static_cast<float*>(nullptr), ws.extremes.ptr, static_cast<float*>(nullptr));
            VB_LAUNCH(kmeans_norms_kernel, norm_blocks, 256, 0, centroids_dev, k, dim, ws.shift.ptr, static_cast<float*>(nullptr),
                      static_cast<float*>(nullptr), static_cast<float*>(nullptr), ws.extremes.ptr, static_cast<float*>(nullptr));
            float top = 0.f;
            VB_CUDA(cudaMemcpyAsync(&top, ws.extremes.ptr, sizeof(float), cudaMemcpyDeviceToHost, st));
            VB_TRY(sync_stream());
            // a power of two that puts the largest element into [2^(top - 1), 2^top); 0: the data do not fit (not finite, or
            // all rows and centroids alike)
            int exponent = 0;
            (void)std::frexp(top, &exponent);
            ws.scale = top > 0.f && top < INFINITY && exponent > -50 && exponent < 50 ? std::ldexp(1.0f, top_exponent - exponent) : 0.f;
            if (ws.scale != 0.f && !ws.half_off) {
                VB_TRY(tc_pretile_f16(x_dev + r0 * dim, rows, dim, ws.shift.ptr, ws.scale, nullptr, ws.x_hi.ptr));
            } else {
                VB_TRY(ws.x_lo.reserve(x_elems));
                VB_TRY(tc_pretile_f32(x_dev + r0 * dim, rows, dim, ws.x_hi.ptr, ws.x_lo.ptr));
            }
            ws.tiled_rows = whole ? x_dev : nullptr;
            ws.tiled_n = whole ? n : 0;
            ws.tiled_dim = dim;
        }
        const bool half = ws.scale != 0.f && !ws.half_off;
        if (!half) {   // split terms of the vectors as they are: the same formulas with no shift
            VB_CUDA(cudaMemsetAsync(ws.shift.ptr, 0, dim * sizeof(float), st));
        }
        VB_CUDA(cudaMemsetAsync(ws.extremes.ptr, 0, 3 * sizeof(float), st));
        VB_LAUNCH(kmeans_norms_kernel, std::min(norm_blocks, (k + 7) / 8), 256, 0, centroids_dev, k, dim, ws.shift.ptr,
                  static_cast<float*>(nullptr), static_cast<float*>(nullptr), ws.c_shifted.ptr, ws.extremes.ptr, ws.extremes.ptr + 1);
        VB_TRY(row_sqnorm_f32(ws.c_shifted.ptr, k, dim, ws.cs_sq.ptr));
        const uint32_t depth = half ? dim + TC_BIAS_DIMS : dim, chunks = (depth + TC_KC - 1) / TC_KC;
        TcOperand a{ws.x_hi.ptr, half ? nullptr : ws.x_lo.ptr, rows, chunks, depth}, b{ws.c_hi.ptr, nullptr, k, chunks, depth};
        if (half) {
            VB_TRY(tc_pretile_f16(centroids_dev, k, dim, ws.shift.ptr, ws.scale, ws.cs_sq.ptr, ws.c_hi.ptr));
        } else {
            VB_TRY(ws.c_lo.reserve(c_elems));
            VB_TRY(tc_pretile_f32(centroids_dev, k, dim, ws.c_hi.ptr, ws.c_lo.ptr));
            b.lo = ws.c_lo.ptr;
        }
        // margins: twice the error of a nominating score, and of the exact chains that decide (2 (dim + 2) 2^-24 each)
        const float chain = 4.0f * static_cast<float>(dim + 8) * 6.0e-8f;
        const float floor_each = half ? std::ldexp(std::sqrt(static_cast<float>(dim)) * 1.001f, -24) * ws.scale : 0.f;
        const float floor = half ? std::ldexp(1.0f, -31) + std::ldexp(static_cast<float>(dim), -49) : 0.f;
        VB_TRY(ws.row_margin.reserve(rows));
        VB_TRY(ws.row_bound.reserve(rows));
        VB_LAUNCH(kmeans_row_prep_kernel, static_cast<uint32_t>((rows * 8 + 255) / 256), 256, 0, x_dev + r0 * dim, rows, dim, ws.shift.ptr,
                  ws.c_shifted.ptr, ws.cs_sq.ptr, k, prev_labels_dev != nullptr ? prev_labels_dev + r0 : nullptr, ws.x_norm.ptr,
                  half ? ws.xs_norm.ptr : ws.x_norm.ptr, ws.extremes.ptr, half ? 4.0e-3f : 1e-3f, chain,
                  half ? static_cast<float>(dim + 16) * 2.4e-7f : 0.f, floor_each, floor, half ? std::ldexp(1.4f, top_exponent) / ws.scale : INFINITY,
                  half ? 0.5f * ws.scale * ws.scale : 1.0f, ws.row_margin.ptr, ws.row_bound.ptr);
        const float* row_bound = prev_labels_dev != nullptr ? ws.row_bound.ptr : nullptr;
        uint32_t n_split = 1, n_flagged = 0;
        VB_TRY(ws.row_flags.reserve(rows));
        VB_CUDA(cudaMemsetAsync(ws.row_flags.ptr, 0, rows * sizeof(uint32_t), st));
        VB_TRY(tc_candidates(ws.tc, a, b, half ? TC_HALF : 3, half ? 1.0f : -2.0f, half ? static_cast<const float*>(nullptr) : ws.cs_sq.ptr, m, 0, ws.cand,
                             &n_split, ws.row_margin.ptr, row_bound, ws.row_flags.ptr, &n_flagged));
        const uint32_t per_row = n_split * m;
        float* best = best_dev != nullptr ? best_dev + r0 : nullptr;
        const uint32_t* close = nullptr;
        if (best == nullptr) {
            VB_TRY(ws.close_rows.reserve(rows + 1));
            VB_CUDA(cudaMemsetAsync(ws.close_rows.ptr, 0, sizeof(uint32_t), st));
            VB_LAUNCH(kmeans_single_kernel, static_cast<uint32_t>((rows * PICK_LANES + 255) / 256), 256, 0, rows, ws.cand.ptr, per_row,
                      ws.row_margin.ptr, labels_dev + r0, ws.close_rows.ptr);
            close = ws.close_rows.ptr;
        }
        const uint32_t pick_blocks = static_cast<uint32_t>(std::min<uint64_t>((rows * PICK_LANES + 255) / 256, 8ull * sm_count()));
        VB_LAUNCH(kmeans_pick_kernel, pick_blocks, 256, 0, x_dev + r0 * dim, rows, dim, centroids_dev, ws.c_sq.ptr, ws.cand.ptr, per_row,
                  ws.row_margin.ptr, close, labels_dev + r0, best);
        if (n_flagged > 0) {
            // A candidate list of these rows ended full of columns within the error margin of its best (many
            // near-equal centroids, or data far from the origin): the exact winner may not have been
            // nominated.  They are decided over all centroids instead.
            VB_TRY(ws.flagged_rows.reserve(n_flagged));
            VB_TRY(ws.flagged_count.reserve(1));
            VB_CUDA(cudaMemsetAsync(ws.flagged_count.ptr, 0, sizeof(uint32_t), st));
            VB_LAUNCH(kmeans_collect_flagged_kernel, static_cast<uint32_t>((rows + 255) / 256), 256, 0, ws.row_flags.ptr,
                      rows, ws.flagged_rows.ptr, ws.flagged_count.ptr);
            const size_t smem = RS_STAGES * RS_STAGE + (dim + 3) / 4 * 4 * sizeof(float);
            if (n_flagged <= KMEANS_FEW_ROWS && smem <= 200 * 1024) {
                VB_TRY(ws.flagged_keys.reserve(n_flagged));
                VB_CUDA(cudaMemsetAsync(ws.flagged_keys.ptr, 0xFF, n_flagged * sizeof(unsigned long long), st));
                auto kernel = dim % 4 == 0 && (reinterpret_cast<uintptr_t>(centroids_dev) & 15) == 0 ? kmeans_few_rows_kernel<16>
                                                                                                     : kmeans_few_rows_kernel<4>;
                VB_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(kernel), smem));
                const uint32_t chunks128 = (k + RS_ROWS - 1) / RS_ROWS;
                const uint32_t shares = std::min(chunks128, std::max(1u, 4u * static_cast<uint32_t>(sm_count()) / n_flagged));
                VB_LAUNCH(kernel, dim3(n_flagged, shares), RS_ROWS, smem, x_dev + r0 * dim, dim, centroids_dev, ws.c_sq.ptr, k,
                          ws.flagged_rows.ptr, ws.flagged_keys.ptr);
                VB_LAUNCH(kmeans_keys_to_labels_kernel, (n_flagged + 255) / 256, 256, 0, ws.flagged_keys.ptr, n_flagged, ws.flagged_rows.ptr,
                          labels_dev + r0, best);
            } else {
                VB_TRY(ws.flagged_x.reserve(static_cast<size_t>(n_flagged) * dim));
                VB_TRY(ws.flagged_labels.reserve(n_flagged));
                VB_TRY(ws.flagged_best.reserve(n_flagged));
                const uint64_t elems = static_cast<uint64_t>(n_flagged) * dim;
                VB_LAUNCH(kmeans_gather_rows_kernel, static_cast<uint32_t>((elems + 255) / 256), 256, 0, x_dev + r0 * dim, dim,
                          ws.flagged_rows.ptr, n_flagged, ws.flagged_x.ptr);
                VB_TRY(dense_argmin_f32(ws.flagged_x.ptr, n_flagged, centroids_dev, k, dim, -2.0f, ws.c_sq.ptr,
                                        ws.flagged_labels.ptr, ws.flagged_best.ptr));
                VB_LAUNCH(kmeans_scatter_labels_kernel, static_cast<uint32_t>((n_flagged + 255) / 256), 256, 0,
                          ws.flagged_rows.ptr, n_flagged, ws.flagged_labels.ptr, ws.flagged_best.ptr, labels_dev + r0,
                          best_dev != nullptr ? best_dev + r0 : nullptr);
            }
            if (half && n_flagged > rows / 16) {
                ws.tiled_rows = nullptr;
                ws.half_off = true;
            }
        }
    }
    return 0;
}

int
kmeans_assign_device(KMeansWorkspace& ws, const float* x_dev, uint64_t n, uint32_t dim,
                     const float* centroids_dev, uint32_t k, int32_t* labels_dev,
                     double* mean_err_host, const int32_t* prev_labels_dev) {
    VB_TRY(ws.c_sq.reserve(k));
    float* best = nullptr;   // wanted for the mean error only
    if (mean_err_host != nullptr) {
        VB_TRY(ws.best.reserve(n));
        best = ws.best.ptr;
    }
    VB_TRY(row_sqnorm_f32(centroids_dev, k, dim, ws.c_sq.ptr));
    if (tensor_cores_enabled() && k >= 64 && n >= 128) {
        VB_TRY(kmeans_assign_tc(ws, x_dev, n, dim, centroids_dev, k, labels_dev, best, prev_labels_dev));
    } else {
        VB_TRY(dense_argmin_f32(x_dev, n, centroids_dev, k, dim, -2.0f, ws.c_sq.ptr, labels_dev, best));
    }
    if (mean_err_host != nullptr) {
        VB_TRY(ws.err.reserve(1));
        VB_CUDA(cudaMemsetAsync(ws.err.ptr, 0, sizeof(double), current_stream()));
        VB_TRY(ws.x_sq.reserve(n));
        VB_TRY(row_sqnorm_f32(x_dev, n, dim, ws.x_sq.ptr));
        VB_LAUNCH(kmeans_error_kernel, static_cast<uint32_t>(std::min<uint64_t>((n + 255) / 256, 4ull * sm_count())), 256, 0, ws.x_sq.ptr, n,
                  ws.best.ptr, ws.err.ptr);
        double total = 0.0;
        VB_CUDA(cudaMemcpyAsync(&total, ws.err.ptr, sizeof(double), cudaMemcpyDeviceToHost,
                                current_stream()));
        VB_TRY(sync_stream());
        *mean_err_host = total / static_cast<double>(static_cast<float>(n));
    }
    return 0;
}

// Centroid sums in a fixed order.  The reference adds the rows of a cluster in 1024-point chunks whose
// partial sums it merges in thread-completion order (kmeans_cluster.cpp:106-172), so its own centroids
// vary from run to run in the last bits.  Here every cluster is summed in ascending row order, one
// fp32 addition per row -- the order the CPU oracle uses -- so training is reproducible bit for bit:
// rows are sorted by (label, row) with a stable radix sort, and one CTA per cluster walks its rows.

// keys[i] = label of row i (k for rows without a valid label), rows[i] = i.
__global__ void
kmeans_sort_keys_kernel(const int32_t* __restrict__ labels, uint64_t n, uint32_t k, uint32_t* __restrict__ keys,
                        uint32_t* __restrict__ rows) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) {
        return;
    }
    const int32_t l = labels[i];
    keys[i] = l >= 0 && static_cast<uint32_t>(l) < k ? static_cast<uint32_t>(l) : k;
    rows[i] = static_cast<uint32_t>(i);
}

// off[j] = number of sorted keys below j, j = 0 .. k.  (Counted while the keys are written, an atomic per row, they took 46 us
// for 1M rows, and the prefix sums another launch.)
__global__ void
kmeans_cluster_offsets_kernel(const uint32_t* __restrict__ keys, uint64_t n, uint32_t k, uint32_t* __restrict__ off) {
    const uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i > n) {
        return;
    }
    const uint32_t here = i < n ? keys[i] : k;
    for (uint32_t j = i > 0 ? keys[i - 1] + 1 : 0u; j <= here; ++j) {
        off[j] = static_cast<uint32_t>(i);
    }
}

// centroids[j][d] = (((x[r0][d] + x[r1][d]) + x[r2][d]) + ...) / count over the rows r0 < r1 < ... of cluster j; a cluster without
// rows takes a row of its own.  One CTA per cluster, one thread per dimension (strided when dim exceeds the CTA).  The time is
// the longest cluster's chain: its row numbers lie in shared memory, the loads of 32 rows are issued together and a batch
// ahead of the additions, which stay in row order (1M x 128 rows in 4096 clusters: 396 us with eight loads together, 335 with 32,
// 240 with the next 32 on their way, 132 with the row numbers at hand and the means formed here).
constexpr uint32_t SUM_ROWS = 1024;   // row numbers in shared memory

__global__ void __launch_bounds__(256, 2)
kmeans_mean_in_order_kernel(const float* __restrict__ x, uint64_t n, uint32_t dim, uint32_t iter, const uint32_t* __restrict__ sorted_rows,
                            const uint32_t* __restrict__ off, int32_t* __restrict__ counts, float* __restrict__ centroids) {
    __shared__ uint32_t row[SUM_ROWS];
    const uint32_t j = blockIdx.x;
    const uint32_t beg = off[j], end = off[j + 1];
    if (threadIdx.x == 0) {
        counts[j] = static_cast<int32_t>(end - beg);
    }
    for (uint32_t d0 = 0; d0 < dim; d0 += blockDim.x) {
        const uint32_t d = d0 + threadIdx.x;
        const bool live = d < dim;
        const float* column = x + (live ? d : 0);
        float s = 0.f;
        for (uint32_t r0 = beg; r0 < end; r0 += SUM_ROWS) {
            const uint32_t m = min(end - r0, SUM_ROWS);
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < m; i += blockDim.x) {
                row[i] = __ldg(sorted_rows + r0 + i);
            }
            __syncthreads();
            uint32_t r = 0;
            if (live && m >= 32) {
                float v[32];
                auto load = [&](float (&w)[32], uint32_t at) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        w[i] = __ldg(column + static_cast<uint64_t>(row[at + i]) * dim);
                    }
                };
                auto add = [&](const float (&w)[32]) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        s = __fadd_rn(s, w[i]);
                    }
                };
                load(v, 0);
                for (; r + 96 <= m; r += 64) {   // a batch is on its way while the one before it is added
                    float w[32];
                    load(w, r + 32);
                    add(v);
                    load(v, r + 64);
                    add(w);
                }
                add(v);
                r += 32;
                if (r + 32 <= m) {
                    load(v, r);
                    add(v);
                    r += 32;
                }
            }
            for (; live && r + 8 <= m; r += 8) {
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    v[i] = __ldg(column + static_cast<uint64_t>(row[r + i]) * dim);
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    s = __fadd_rn(s, v[i]);
                }
            }
            for (; live && r < m; ++r) {
                s = __fadd_rn(s, __ldg(column + static_cast<uint64_t>(row[r]) * dim));
            }
        }
        if (live) {
            if (end > beg) {
                s = __fmul_rn(s, __fdiv_rn(1.0f, static_cast<float>(static_cast<int32_t>(end - beg))));
            } else {
                s = column[(static_cast<uint64_t>(j) * 2654435761ull + iter) % n * dim];
            }
            centroids[static_cast<uint64_t>(j) * dim + d] = s;
        }
    }
}

int
kmeans_update_device(KMeansWorkspace& ws, const float* x_dev, uint64_t n, uint32_t dim,
                     const int32_t* labels_dev, uint32_t k, uint32_t iter, float* centroids_dev) {
    VB_CHECK_ARG(n < 0xFFFFFFFFull, "kmeans update: batch too large");
    VB_TRY(ws.counts.reserve(k));
    VB_TRY(ws.sort_keys_in.reserve(n));
    VB_TRY(ws.sort_keys_out.reserve(n));
    VB_TRY(ws.sort_rows_in.reserve(n));
    VB_TRY(ws.sort_rows_out.reserve(n));
    VB_TRY(ws.cluster_off.reserve(static_cast<size_t>(k) + 1));
    cudaStream_t st = current_stream();
    VB_LAUNCH(kmeans_sort_keys_kernel, static_cast<uint32_t>((n + 255) / 256), 256, 0, labels_dev, n, k,
              ws.sort_keys_in.ptr, ws.sort_rows_in.ptr);
    {
        // stable sort by label: rows of a cluster stay in ascending order
        int end_bit = 1;
        while ((uint64_t{1} << end_bit) <= k) {
            ++end_bit;
        }
        size_t tmp_bytes = 0;
        VB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, ws.sort_keys_in.ptr, ws.sort_keys_out.ptr,
                                                ws.sort_rows_in.ptr, ws.sort_rows_out.ptr, static_cast<int64_t>(n), 0,
                                                end_bit, st));
        VB_TRY(ws.sort_tmp.reserve(tmp_bytes > 0 ? tmp_bytes : 1));
        tmp_bytes = ws.sort_tmp.cap;
        VB_CUDA(cub::DeviceRadixSort::SortPairs(ws.sort_tmp.ptr, tmp_bytes, ws.sort_keys_in.ptr, ws.sort_keys_out.ptr,
                                                ws.sort_rows_in.ptr, ws.sort_rows_out.ptr, static_cast<int64_t>(n), 0,
                                                end_bit, st));
        g_kernel_launches.fetch_add(1);
    }
    VB_LAUNCH(kmeans_cluster_offsets_kernel, static_cast<uint32_t>(n / 256 + 1), 256, 0, ws.sort_keys_out.ptr, n, k, ws.cluster_off.ptr);
    // (threads for the dimensions there are: the more CTAs of few dimensions an SM holds, the more rows are on their way)
    VB_LAUNCH(kmeans_mean_in_order_kernel, k, dim <= 224 ? (dim + 31) / 32 * 32 : 256, 0, x_dev, n, dim, iter, ws.sort_rows_out.ptr,
              ws.cluster_off.ptr, ws.counts.ptr, centroids_dev);
    return 0;
}

}  // namespace vb200

using namespace vb200;

// The training entry points keep one workspace per process between calls (tiled rows, candidate lists, sort
// buffers: 1.3 GB for 1 M x 128 rows against 4096 centroids), because allocating and freeing it costs more than
// two Lloyd iterations; a second caller at the same time gets a workspace of its own.
// vb200_release_workspaces() frees the kept one.
namespace {

std::mutex g_kmeans_ws_mu;
KMeansWorkspace* g_kmeans_ws = nullptr;   // never destroyed at exit: the CUDA context may be gone by then

class WorkspaceLease {
public:
    WorkspaceLease() : kept_(g_kmeans_ws_mu.try_lock()) {
        if (kept_ && g_kmeans_ws == nullptr) {
            g_kmeans_ws = new (std::nothrow) KMeansWorkspace;
            if (g_kmeans_ws == nullptr) {
                g_kmeans_ws_mu.unlock();
                kept_ = false;
            }
        }
        if (kept_) {
            g_kmeans_ws->forget_points();   // another call's rows may have lived at the same address
        }
    }
    ~WorkspaceLease() {
        if (kept_) {
            g_kmeans_ws_mu.unlock();
        }
    }
    KMeansWorkspace& get() { return kept_ ? *g_kmeans_ws : own_; }

private:
    bool kept_;
    KMeansWorkspace own_;
};

}  // namespace

extern "C" int
vb200_release_workspaces(void) {
    std::lock_guard<std::mutex> lock(g_kmeans_ws_mu);
    ReleaseScope scope;
    delete g_kmeans_ws;
    g_kmeans_ws = nullptr;
    (void)sync_stream();   // what was freed is free now
    pool_trim();
    return 0;
}

static int
check_kmeans_args(const float* data, uint64_t count, uint32_t dim, const float* centroids, uint32_t k) {
    // Argument checks of KMeansCluster::Run (kmeans_cluster.cpp:54-65).
    VB_CHECK_ARG(k > 0, "k must be positive");
    VB_CHECK_ARG(count > 0, "count must be positive");
    VB_CHECK_ARG(data != nullptr, "datas cannot be null");
    VB_CHECK_ARG(dim > 0, "dim must be positive");
    VB_CHECK_ARG(centroids != nullptr, "centroids cannot be null");
    return 0;
}

extern "C" int
vb200_kmeans_assign(const float* data, uint64_t count, uint32_t dim, const float* centroids,
                    uint32_t k, int32_t* labels, double* mean_err) {
    VB_TRY(check_kmeans_args(data, count, dim, centroids, k));
    VB_CHECK_ARG(labels != nullptr, "labels cannot be null");
    DevInput<float> x, c;
    VB_TRY(x.bind(data, count * dim));
    VB_TRY(c.bind(centroids, static_cast<size_t>(k) * dim));
    DevBuf<int32_t> lab;
    VB_TRY(lab.reserve(count));
    KMeansWorkspace ws;
    VB_TRY(kmeans_assign_device(ws, x.ptr, count, dim, c.ptr, k, lab.ptr, mean_err));
    VB_TRY(copy_out(labels, lab.ptr, count));
    return sync_stream();
}

extern "C" int
vb200_kmeans_update(const float* data, uint64_t count, uint32_t dim, const int32_t* labels,
                    uint32_t k, uint32_t iter, float* centroids, int32_t* counts) {
    VB_TRY(check_kmeans_args(data, count, dim, centroids, k));
    VB_CHECK_ARG(labels != nullptr, "labels cannot be null");
    DevInput<float> x;
    DevInput<int32_t> lab;
    VB_TRY(x.bind(data, count * dim));
    VB_TRY(lab.bind(labels, count));
    DevBuf<float> c;
    VB_TRY(c.reserve(static_cast<size_t>(k) * dim));
    KMeansWorkspace ws;
    VB_TRY(kmeans_update_device(ws, x.ptr, count, dim, lab.ptr, k, iter, c.ptr));
    VB_TRY(copy_out(centroids, c.ptr, static_cast<size_t>(k) * dim));
    if (counts != nullptr) {
        VB_TRY(copy_out(counts, ws.counts.ptr, k));
    }
    return sync_stream();
}

extern "C" int
vb200_kmeans_train(const float* data, uint64_t count, uint32_t dim, uint32_t k, int iters,
                   float* centroids, int32_t* labels, double* mean_err) {
    VB_TRY(check_kmeans_args(data, count, dim, centroids, k));
    VB_CHECK_ARG(k <= count, "k cannot be larger than count");
    VB_CHECK_ARG(iters >= 0, "iters must not be negative");
    DevInput<float> x;
    VB_TRY(x.bind(data, count * dim));
    const size_t kd = static_cast<size_t>(k) * dim;
    DevBuf<float> c;
    VB_TRY(c.reserve(kd));
    VB_CUDA(cudaMemcpyAsync(c.ptr, centroids, kd * sizeof(float), cudaMemcpyDefault, current_stream()));
    DevBuf<int32_t> lab;
    VB_TRY(lab.reserve(count));
    WorkspaceLease lease;
    KMeansWorkspace& ws = lease.get();
    for (int it = 0; it < iters; ++it) {
        double* err = (it == iters - 1) ? mean_err : nullptr;
        VB_TRY(kmeans_assign_device(ws, x.ptr, count, dim, c.ptr, k, lab.ptr, err, it > 0 ? lab.ptr : nullptr));
        VB_TRY(kmeans_update_device(ws, x.ptr, count, dim, lab.ptr, k, static_cast<uint32_t>(it), c.ptr));
    }
    VB_TRY(copy_out(centroids, c.ptr, kd));
    if (labels != nullptr && iters > 0) {
        VB_TRY(copy_out(labels, lab.ptr, count));
    }
    return sync_stream();
}

// ---------------------------------------------------------------------------------------------
// k-means++ seeding (KMeansCluster::select_initial_centroids_kmeans_plus_plus,
// src/impl/cluster/kmeans_cluster.cpp:383-435)
// ---------------------------------------------------------------------------------------------
namespace vb200 {

constexpr uint32_t KPP_BLOCK_ROWS = 1024;   // rows per CTA of the update kernel = one partial sum

// min_d[i] = min(min_d[i], |x_i - c|^2) with the reference's per-row chain (difference, then one
// FMA per dimension in ascending order); part[b] = sum of the CTA's rows in double.  A warp
// stages 32 rows x 32 dimensions through shared memory so the global reads stay coalesced while
// every lane still walks its own row in order.
__global__ void __launch_bounds__(256)
kpp_update_kernel(const float* __restrict__ x, uint64_t n, uint32_t dim, const float* __restrict__ centroid,
                  float* __restrict__ min_d, double* __restrict__ part) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* c = reinterpret_cast<float*>(smem_raw);                       // dim
    float* tiles = c + ((dim + 31) / 32) * 32;                            // 8 warps x 32 x 33
    __shared__ double warp_sum[8];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t d = threadIdx.x; d < dim; d += blockDim.x) {
        c[d] = centroid[d];
    }
    __syncthreads();
    float* tile = tiles + warp * (32 * 33);
    double acc = 0.0;
    const uint64_t block_row0 = static_cast<uint64_t>(blockIdx.x) * KPP_BLOCK_ROWS;
    for (uint32_t pass = 0; pass < KPP_BLOCK_ROWS / 256; ++pass) {
        const uint64_t row0 = block_row0 + (pass * 8 + warp) * 32;
        if (row0 >= n) {
            break;
        }
        float s = 0.f;
        for (uint32_t d0 = 0; d0 < dim; d0 += 32) {
            __syncwarp();
            for (uint32_t r = 0; r < 32; ++r) {
                const uint64_t row = row0 + r;
                const uint32_t d = d0 + lane;
                tile[r * 33 + lane] = (row < n && d < dim) ? __ldg(x + row * dim + d) : 0.f;
            }
            __syncwarp();
            const uint32_t lim = dim - d0 < 32 ? dim - d0 : 32;
            for (uint32_t j = 0; j < lim; ++j) {
                const float t = __fsub_rn(tile[lane * 33 + j], c[d0 + j]);
                s = fmaf(t, t, s);
            }
        }
        const uint64_t row = row0 + lane;
        if (row < n) {
            const float old = min_d[row];
            const float m = s < old ? s : old;
            min_d[row] = m;
            acc += static_cast<double>(m);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        acc += __shfl_xor_sync(0xffffffffu, acc, o);
    }
    if (lane == 0) {
        warp_sum[warp] = acc;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < 8; ++w) {
            t += warp_sum[w];
        }
        part[blockIdx.x] = t;
    }
}

// One CTA: total of the partial sums; threshold = total * u (the uniform draw from [0, total));
// the first row whose running sum reaches it becomes centroid `slot`.  With total <= 0 (every row
// coincides with a chosen centre) nothing is picked and the round is recorded in state[0]; the
// host then finishes the seeding with uniform draws as the reference does.
__global__ void __launch_bounds__(1024)
kpp_pick_kernel(const float* __restrict__ x, uint64_t n, uint32_t dim, const float* __restrict__ min_d,
                const double* __restrict__ part, uint32_t n_part, double u, uint32_t slot,
                float* __restrict__ centroids, int64_t* __restrict__ picked, uint32_t* __restrict__ state) {
    __shared__ double sh_scan[1024];
    __shared__ double sh_base;
    __shared__ uint32_t sh_block;
    __shared__ unsigned long long sh_row;
    const uint32_t t = threadIdx.x;
    // inclusive scan of the partial sums, each thread owning a contiguous run
    const uint32_t per = (n_part + 1023) / 1024;
    const uint32_t p0 = t * per;
    double local = 0.0;
    for (uint32_t i = p0; i < p0 + per && i < n_part; ++i) {
        local += part[i];
    }
    sh_scan[t] = local;
    __syncthreads();
    for (uint32_t off = 1; off < 1024; off <<= 1) {
        double v = t >= off ? sh_scan[t - off] : 0.0;
        __syncthreads();
        sh_scan[t] += v;
        __syncthreads();
    }
    const double total = sh_scan[1023];
    if (!(total > 0.0)) {
        if (t == 0) {
            atomicMin(state, slot);
        }
        return;
    }
    const double thr = total * u + 0.0;
    if (t == 0) {
        sh_block = 0xFFFFFFFFu;
        sh_row = ~0ull;
    }
    __syncthreads();
    // first run, then first partial sum inside it, whose inclusive sum reaches the threshold
    const double before = t > 0 ? sh_scan[t - 1] : 0.0;
    if (sh_scan[t] >= thr && !(before >= thr) && p0 < n_part) {
        const uint32_t last = p0 + per - 1 < n_part ? p0 + per - 1 : n_part - 1;
        double run = before;
        for (uint32_t i = p0; i <= last; ++i) {
            const double next = run + part[i];
            if (next >= thr || i == last) {
                sh_block = i;
                sh_base = run;
                break;
            }
            run = next;
        }
    }
    __syncthreads();
    uint64_t row_pick = n - 1;   // the reference's default when the running sum never gets there
    if (sh_block != 0xFFFFFFFFu) {
        const uint64_t row0 = static_cast<uint64_t>(sh_block) * KPP_BLOCK_ROWS;
        const uint64_t row = row0 + t;
        const double base = sh_base;
        __syncthreads();
        sh_scan[t] = row < n ? static_cast<double>(min_d[row]) : 0.0;
        __syncthreads();
        for (uint32_t off = 1; off < 1024; off <<= 1) {
            double v = t >= off ? sh_scan[t - off] : 0.0;
            __syncthreads();
            sh_scan[t] += v;
            __syncthreads();
        }
        if (row < n && base + sh_scan[t] >= thr) {
            atomicMin(&sh_row, static_cast<unsigned long long>(row));
        }
        __syncthreads();
        if (sh_row != ~0ull) {
            row_pick = sh_row;
        } else {
            // rounding kept the CTA's own running sum just below the threshold: its last row
            const uint64_t last = row0 + KPP_BLOCK_ROWS - 1;
            row_pick = last < n ? last : n - 1;
        }
    }
    for (uint32_t d = t; d < dim; d += blockDim.x) {
        centroids[static_cast<uint64_t>(slot) * dim + d] = x[row_pick * dim + d];
    }
    if (t == 0 && picked != nullptr) {
        picked[slot] = static_cast<int64_t>(row_pick);
    }
}

__global__ void
kpp_fill_kernel(float* __restrict__ min_d, uint64_t n, uint32_t* __restrict__ state) {
    uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) {
        min_d[i] = 3.402823466e+38f;
    }
    if (i == 0) {
        state[0] = 0xFFFFFFFFu;
    }
}

__global__ void
kpp_copy_row_kernel(const float* __restrict__ x, uint64_t row, uint32_t dim, uint32_t slot,
                    float* __restrict__ centroids, int64_t* __restrict__ picked) {
    for (uint32_t d = threadIdx.x; d < dim; d += blockDim.x) {
        centroids[static_cast<uint64_t>(slot) * dim + d] = x[row * dim + d];
    }
    if (threadIdx.x == 0 && picked != nullptr) {
        picked[slot] = static_cast<int64_t>(row);
    }
}

// All rounds as one cooperative launch (kpp.cuh).  *done = false when the device cannot hold the grid (an SM limit on
// the context): the caller then seeds round by round.
static int
kpp_run_rounds(const float* x_dev, uint64_t n, uint32_t dim, uint32_t k, uint64_t first, const std::vector<double>& u, float* min_d,
               uint32_t* state, float* centroids_dev, int64_t* picked_dev, bool* done) {
    *done = false;
    const uint32_t sms = static_cast<uint32_t>(sm_count());
    const uint64_t resident_per = std::max<uint64_t>((n + sms - 1) / sms, 16);
    constexpr int THREADS = 512;
    // dimensions of a row in registers, where each row of a CTA has a thread (80 is what 128 registers a thread have room for)
    const uint32_t reg = resident_per <= THREADS ? (dim <= 32 ? 32u : (dim <= 64 ? 64u : 80u)) : 0u;
    const size_t qpad = std::max<size_t>((dim + 3) / 4 * 4, reg);
    // rows per CTA when every SM takes a share (at least 16 rows: fewer are not worth a CTA in the barriers)
    const size_t resident_bytes = (qpad + resident_per * ((dim | 1u) + 1)) * sizeof(float);
    const bool resident = resident_bytes <= 216 * 1024;
    const bool wide = dim % 4 == 0 && (reinterpret_cast<uintptr_t>(x_dev) & 15) == 0;
    const size_t smem = resident ? resident_bytes : RS_STAGES * RS_STAGE + (dim + 3) / 4 * 4 * sizeof(float);
    if (smem > 216 * 1024) {
        return 0;
    }
    const void* kernel = nullptr;
    if (resident) {
        kernel = reg == 32 ? reinterpret_cast<const void*>(kpp_rounds_kernel<true, 32, 4, THREADS>)
                           : (reg == 64 ? reinterpret_cast<const void*>(kpp_rounds_kernel<true, 64, 4, THREADS>)
                                        : (reg == 80 ? reinterpret_cast<const void*>(kpp_rounds_kernel<true, 80, 4, THREADS>)
                                                     : reinterpret_cast<const void*>(kpp_rounds_kernel<true, 0, 4, THREADS>)));
    } else {
        kernel = wide ? reinterpret_cast<const void*>(kpp_rounds_kernel<false, 0, 16, RS_ROWS>)
                      : reinterpret_cast<const void*>(kpp_rounds_kernel<false, 0, 4, RS_ROWS>);
    }
    const int threads = resident ? THREADS : RS_ROWS;
    VB_TRY(allow_dynamic_smem(kernel, smem));
    int per_sm = 0;
    VB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    if (per_sm < 1) {
        return 0;
    }
    KppRounds p{};
    p.x = x_dev;
    p.n = n;
    p.dim = dim;
    p.k = k;
    if (resident) {
        p.per = resident_per;
    } else {
        const uint64_t most = std::min<uint64_t>(std::min<uint64_t>(static_cast<uint64_t>(sms) * per_sm, RS_ROWS * KPP_RUN), (n + RS_ROWS - 1) / RS_ROWS);
        p.per = (n + most - 1) / most;
    }
    const uint64_t grid = (n + p.per - 1) / p.per;
    if (grid > (resident ? 32 : RS_ROWS) * KPP_RUN || (!resident && n > 0xFFFFFFFFull)) {   // (a row's number is a word of 32 bits)
        return 0;
    }
    p.first = first;
    DevBuf<double> draws;
    DevBuf<unsigned long long> words;   // the sums' two sets, the row's, whether a wait gave up, and the sums' count
    const size_t n_words = 4 * grid + dim + 2;
    VB_TRY(draws.reserve(k));
    VB_TRY(words.reserve(n_words));
    VB_CUDA(cudaMemsetAsync(words.ptr, 0, n_words * sizeof(unsigned long long), current_stream()));
    VB_CUDA(cudaMemcpyAsync(draws.ptr, u.data(), k * sizeof(double), cudaMemcpyHostToDevice, current_stream()));
    p.u = draws.ptr;
    p.min_d = min_d;
    p.part = words.ptr;
    p.row = words.ptr + 4 * grid;
    p.failed = reinterpret_cast<uint32_t*>(words.ptr + 4 * grid + dim);
    p.count = words.ptr + 4 * grid + dim + 1;
    p.spin_limit = tc_spin_limit();
    p.centroids = centroids_dev;
    p.picked = picked_dev;
    p.state = state;
    void* args[] = {&p};
    const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(static_cast<uint32_t>(grid)), dim3(threads), args, smem, current_stream());
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported) {
        (void)cudaGetLastError();
        return 0;
    }
    VB_CUDA(e);
    g_kernel_launches.fetch_add(1, std::memory_order_relaxed);
    uint32_t failed = 0;
    VB_CUDA(cudaMemcpyAsync(&failed, p.failed, sizeof(failed), cudaMemcpyDeviceToHost, current_stream()));
    VB_TRY(sync_stream());   // (the draws are the caller's)
    if (failed != 0) {
        VB_FAIL(VB200_INTERNAL_ERROR, "the seeding kernel gave up on a bounded wait");
    }
    *done = true;
    return 0;
}

// centroids_dev[k x dim] and (optionally) picked_dev[k] on the device.  The generator and its
// distributions are the C++ library's, exactly the objects the reference draws from; only the
// seed is the caller's (the reference takes it from std::random_device).
int
kmeans_pp_init_device(const float* x_dev, uint64_t n, uint32_t dim, uint32_t k, uint32_t seed,
                      float* centroids_dev, int64_t* picked_dev) {
    VB_CHECK_ARG(n > 0 && k > 0 && k <= n, "k cannot be larger than count");
    const uint32_t n_part = static_cast<uint32_t>((n + KPP_BLOCK_ROWS - 1) / KPP_BLOCK_ROWS);
    DevBuf<float> min_d;
    DevBuf<double> part;
    DevBuf<uint32_t> state;
    VB_TRY(min_d.reserve(n));
    VB_TRY(part.reserve(n_part));
    VB_TRY(state.reserve(1));
    VB_LAUNCH(kpp_fill_kernel, static_cast<uint32_t>((n + 255) / 256), 256, 0, min_d.ptr, n, state.ptr);
    std::mt19937 gen(seed);
    std::uniform_int_distribution<uint64_t> any_row(0, n - 1);
    const uint64_t first = any_row(gen);
    std::uniform_real_distribution<double> unit(0.0, 1.0);
    std::vector<double> u(k, 0.0);
    for (uint32_t c = 1; c < k; ++c) {
        u[c] = unit(gen);
    }
    bool done = false;
    VB_TRY(kpp_run_rounds(x_dev, n, dim, k, first, u, min_d.ptr, state.ptr, centroids_dev, picked_dev, &done));
    if (!done) {
        VB_LAUNCH(kpp_copy_row_kernel, 1, 128, 0, x_dev, first, dim, 0u, centroids_dev, picked_dev);
        const size_t smem = (static_cast<size_t>((dim + 31) / 32) * 32 + 8 * 32 * 33) * sizeof(float);
        VB_CHECK_ARG(smem <= 200 * 1024, "dim too large for the seeding kernel");
        VB_TRY(allow_dynamic_smem(reinterpret_cast<const void*>(kpp_update_kernel), smem));
        for (uint32_t c = 1; c < k; ++c) {
            VB_LAUNCH(kpp_update_kernel, n_part, 256, smem, x_dev, n, dim,
                      centroids_dev + static_cast<size_t>(c - 1) * dim, min_d.ptr, part.ptr);
            VB_LAUNCH(kpp_pick_kernel, 1, 1024, 0, x_dev, n, dim, min_d.ptr, part.ptr, n_part, u[c], c,
                      centroids_dev, picked_dev, state.ptr);
        }
    }
    uint32_t first_flat = 0xFFFFFFFFu;
    VB_CUDA(cudaMemcpyAsync(&first_flat, state.ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, current_stream()));
    VB_TRY(sync_stream());
    if (first_flat < k) {
        // From that round on every row coincides with a chosen centre, so the total stays zero and
        // the reference draws a uniform row each round.  Replay the generator up to there (each
        // earlier round consumed one real draw) and finish the same way.
        std::mt19937 replay(seed);
        (void)any_row(replay);
        for (uint32_t c = 1; c < first_flat; ++c) {
            (void)unit(replay);
        }
        for (uint32_t c = first_flat; c < k; ++c) {
            VB_LAUNCH(kpp_copy_row_kernel, 1, 128, 0, x_dev, any_row(replay), dim, c, centroids_dev, picked_dev);
        }
        VB_TRY(sync_stream());
    }
    return 0;
}

}  // namespace vb200

extern "C" int
vb200_kmeans_init(const float* data, uint64_t count, uint32_t dim, uint32_t k, uint32_t seed, float* centroids,
                  int64_t* picked) {
    VB_TRY(check_kmeans_args(data, count, dim, centroids, k));
    VB_CHECK_ARG(k <= count, "k cannot be larger than count");
    DevInput<float> x;
    VB_TRY(x.bind(data, count * dim));
    DevBuf<float> c;
    DevBuf<int64_t> rows;
    VB_TRY(c.reserve(static_cast<size_t>(k) * dim));
    VB_TRY(rows.reserve(k));
    VB_TRY(kmeans_pp_init_device(x.ptr, count, dim, k, seed, c.ptr, rows.ptr));
    VB_TRY(copy_out(centroids, c.ptr, static_cast<size_t>(k) * dim));
    if (picked != nullptr) {
        VB_TRY(copy_out(picked, rows.ptr, k));
    }
    return sync_stream();
}

// ---------------------------------------------------------------------------------------------
// Assignment without any allocation
// ---------------------------------------------------------------------------------------------
// Some callers must not reach the CUDA allocator at all: a serving thread that holds a fixed
// memory budget and cannot tolerate the device-wide synchronisation cudaMalloc/cudaFree imply, or
// a host that has handed all remaining device memory to another pool.  For them the centroid
// norms -- the only scratch the assignment needs -- live in this fixed array, which every GPU that
// loads the library holds (256 KiB) until the process exits.
constexpr uint32_t NOALLOC_MAX_K = 65536;
static __device__ __align__(256) float g_noalloc_centroid_sq[NOALLOC_MAX_K];

// Device address of the array above, looked up once per device with that device current.  In host
// code the symbol itself is only a stand-in; kernels must be given the address this returns.
static int
noalloc_scratch(float** out) {
    static std::mutex mu;
    static float* cached[64] = {nullptr};
    int dev = 0;
    VB_CUDA(cudaGetDevice(&dev));
    VB_CHECK_ARG(dev >= 0 && dev < 64, "device ordinal %d out of range", dev);
    std::lock_guard<std::mutex> lock(mu);
    if (cached[dev] == nullptr) {
        void* p = nullptr;
        VB_CUDA(cudaGetSymbolAddress(&p, g_noalloc_centroid_sq));
        cached[dev] = static_cast<float*>(p);
    }
    *out = cached[dev];
    return 0;
}

extern "C" int
vb200_kmeans_assign_noalloc(const float* data_dev, uint64_t count, uint32_t dim,
                            const float* centroids_dev, uint32_t k, int32_t* labels_dev) {
    VB_TRY(check_kmeans_args(data_dev, count, dim, centroids_dev, k));
    VB_CHECK_ARG(labels_dev != nullptr, "labels cannot be null");
    VB_CHECK_ARG(k <= NOALLOC_MAX_K, "k = %u exceeds the %u centroids the fixed scratch array holds", k,
                 NOALLOC_MAX_K);
    VB_CHECK_ARG(is_device_pointer(data_dev) && is_device_pointer(centroids_dev) &&
                     is_device_pointer(labels_dev),
                 "this entry point stages nothing: data, centroids and labels must be device pointers");
    // the scratch array used below is the current device's copy
    VB_CHECK_ARG(is_pointer_on_current_device(data_dev) && is_pointer_on_current_device(centroids_dev) &&
                     is_pointer_on_current_device(labels_dev),
                 "data, centroids and labels must live on the device that is current on the calling thread");
    float* c_sq = nullptr;
    VB_TRY(noalloc_scratch(&c_sq));
    // Every call rewrites entries [0, k) before reading them, so nothing has to be cleared.
    VB_TRY(row_sqnorm_f32(centroids_dev, k, dim, c_sq));
    VB_TRY(dense_argmin_f32(data_dev, count, centroids_dev, k, dim, -2.0f, c_sq, labels_dev, nullptr));
    return sync_stream();
}

extern "C" int
vb200_debug_set_wait_limit(int32_t polls) {
    tc_set_spin_limit(polls < 0 ? TC_SPIN_LIMIT : static_cast<uint32_t>(polls));
    return 0;
}

extern "C" int
vb200_set_tensor_cores(int enable) {
    g_tc_enabled.store(enable != 0 ? 1 : 0);
    return 0;
}
