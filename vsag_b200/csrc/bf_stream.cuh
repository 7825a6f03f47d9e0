// Exact search for a few queries: one pass over the rows, a thread per row (row_scan.cuh), the k best kept per CTA.
//
// The bound is the pass over the rows: 1M x 128 fp32 is 512 MB, 78 us at the measured copy rate.  Each distance is
// the reference's chain over ascending dimensions, so what the CTAs keep is final.  Up to eight queries share the
// pass (about 10 instructions per 16 row bytes and query keep it below the memory's time); a tensor-core tile of
// 128 query rows would be mostly empty there.
#pragma once

#include "block_select.cuh"
#include "row_scan.cuh"

namespace vb200 {

constexpr int BF_STREAM_QUERIES = 8;

struct BfStream {
    const void* queries;        // [.. x dim] fp32, or bf16 bit patterns
    const uint32_t* pick;       // [nq] the queries' rows in `queries`, or null: 0 .. nq - 1
    uint32_t nq, dim;
    const unsigned char* base;  // [n x dim] rows in the index's type
    uint64_t n;
    uint32_t k, cap;            // results per query; per-CTA candidate buffer (a power of two >= k + 128)
    uint32_t* bound;            // [nq] ordered value of some query's k-th best so far, 0xFFFFFFFF = none
    uint64_t* part;             // [nq][grid][k]
    const float* masked;        // [n] +inf for rows that are removed or filtered out, or null
};

template <int FMT, bool L2, int QN, int UNIT>
__global__ void __launch_bounds__(RS_ROWS)
bf_stream_kernel(const BfStream p) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr uint32_t ELEM = FMT == ROW_F32 ? 4 : 2;
    const uint32_t qpad = (p.dim + 7) / 8 * 8;
    float* qs = reinterpret_cast<float*>(smem + RS_STAGES * RS_STAGE);
    TileSelect<QN> ts;
    float* unused;
    tile_carve<QN>(reinterpret_cast<unsigned char*>(qs + QN * qpad), p.cap, 0, unused, ts);
    ts.k = p.k;
    ts.cap = p.cap;
    const uint32_t q0 = blockIdx.y * QN;
    const int here = static_cast<int>(p.nq - q0 < QN ? p.nq - q0 : QN);
    for (uint32_t i = threadIdx.x; i < QN * qpad; i += RS_ROWS) {
        const uint32_t qi = i / qpad, d = i - qi * qpad;
        float v = 0.f;
        if (static_cast<int>(qi) < here && d < p.dim) {
            const uint64_t at = static_cast<uint64_t>(p.pick != nullptr ? __ldg(p.pick + q0 + qi) : q0 + qi) * p.dim + d;
            v = FMT == ROW_F32 ? static_cast<const float*>(p.queries)[at]
                               : half_decode<SCAN_FMT_BF16>(static_cast<const uint16_t*>(p.queries)[at]);
        }
        qs[i] = v;
    }
    if (threadIdx.x < QN) {
        const int qi = threadIdx.x;
        ts.cnt[qi] = 0;
        ts.qa[qi] = 0.f;
        ts.qidx[qi] = q0 + qi;
        ts.slot[qi] = (q0 + qi) * gridDim.x + blockIdx.x;
        ts.set_bound(qi, qi < here ? 0xFFFFFFFFu : 0u);
    }
    __syncthreads();
    uint32_t rounds = 0;
    RowAcc<FMT, L2, QN> acc;
    row_stream<UNIT>(p.base, static_cast<uint64_t>(p.dim) * ELEM, p.dim * ELEM, p.dim, p.n, blockIdx.x, gridDim.x, smem, qs, qpad, acc,
                     [&](uint64_t row, bool valid) {
                         if (valid) {
#pragma unroll
                             for (int i = 0; i < QN; ++i) {
                                 if (i < here) {
                                     const float v = L2 ? acc.acc[i] : __fsub_rn(1.0f, acc.acc[i]);
                                     if (v <= ts.thrq[i] && (p.masked == nullptr || __ldg(p.masked + row) < INFINITY)) {
                                         ts.push(i, v, static_cast<uint32_t>(row));
                                     }
                                 }
                             }
                         }
                         __syncthreads();
                         ts.make_room(here);
                         __syncthreads();
                         // every now and then the bounds of the CTAs meet
                         if ((rounds++ & 7u) == 7u) {
                             if (static_cast<int>(threadIdx.x) < here) {
                                 const int qi = threadIdx.x;
                                 const uint32_t mine = ts.thr[qi];
                                 const uint32_t u = mine < 0xFF800000u ? atomicMin(p.bound + q0 + qi, mine)
                                                                       : *reinterpret_cast<volatile uint32_t*>(p.bound + q0 + qi);
                                 if (u < mine) {
                                     ts.set_bound(qi, u);
                                 }
                             }
                             __syncthreads();
                         }
                     });
    __syncthreads();
    ts.finish(here, p.part, p.bound);
}

// One CTA per query: the `keep` best of its `n` partial keys (payload = row), as the first of the k results of query
// pick[blockIdx.x] (null: its own number).
template <int T>
__global__ void __launch_bounds__(T)
bf_pick_kernel(const uint64_t* __restrict__ part, uint32_t n, uint32_t keep, uint32_t k, const uint32_t* __restrict__ pick,
               const int64_t* __restrict__ labels, int64_t* __restrict__ ids, float* __restrict__ dists) {
    __shared__ SelectScratch sel;
    __shared__ __align__(16) uint64_t keys[SELECT_CAP];
    __shared__ __align__(16) uint64_t best[1024];
    const uint64_t* mine = part + static_cast<uint64_t>(blockIdx.x) * n;
    const uint32_t found = block_select<T>(load_source([&](uint32_t i) { return static_cast<uint32_t>(__ldg(mine + i) >> 32); }),
                                           [&](uint32_t i) { return static_cast<uint32_t>(__ldg(mine + i)); }, n, keep, keys, sel);
    block_sort_to<T>(keys, found, keep, best);
    const uint64_t q = pick != nullptr ? __ldg(pick + blockIdx.x) : blockIdx.x;
    for (uint32_t i = threadIdx.x; i < k; i += T) {
        const bool there = i < min(found, keep);
        ids[q * k + i] = there ? __ldg(labels + static_cast<uint32_t>(best[i])) : -1;
        dists[q * k + i] = there ? ordered_to_float(static_cast<uint32_t>(best[i] >> 32)) : INFINITY;
    }
}

// *top = the largest norm of the rows whose squared norms are given, rounded up (one launch per add; never lowered).
__global__ void __launch_bounds__(256)
bf_row_max_kernel(const float* __restrict__ sq, uint64_t n, float* __restrict__ top) {
    float most = 0.f;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x; i < n; i += static_cast<uint64_t>(gridDim.x) * 256) {
        most = fmaxf(most, __ldg(sq + i));
    }
    for (int o = 16; o > 0; o >>= 1) {
        most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
    }
    if ((threadIdx.x & 31) == 0) {   // non-negative floats order like their bit patterns
        atomicMax(reinterpret_cast<int*>(top), __float_as_int(sqrtf(most) * 1.001f));
    }
}

// How far a nominating score may be from the distance it stands for, so that a query knows whether a row that was not
// nominated can belong to its results.  With X = the largest |x| and Q = |q|:
//   IP  the score -<x, q> and the exact 1 - <x, q> differ by (chain + matrix) X Q and the rounding of the subtraction
//   L2  |x|^2 - 2 <x, q> + |q|^2 and the exact chain differ by chain (X^2 + Q^2 + d) + 2 matrix X Q, d the distance
// chain = the rounding of a sum of dim products in fp32, (dim + 16) 2^-24; matrix = that of the tensor cores' sums.  Those
// take 16 products and the running sum per step, each cut one bit below fp32's last or lower: at most (17/16) dim 2^-24 per
// term pair; with split terms three pairs and the dropped products, 3 * 2^-18.
struct BfMargin {
    const float* row_max;   // X
    float chain, matrix;
    uint32_t* unsure;       // [0] = number of queries whose nominations may not be enough, then their numbers
    uint32_t q_base;        // number of the launch's first query
    __device__ __forceinline__ float
    of(bool l2, float top, float qq, float kth) const {
        const float size = top * sqrtf(qq);
        const float margin = l2 ? fmaf(chain, top * top + qq + kth, 2.0f * matrix * size) : fmaf(chain + matrix, size, 3e-7f);
        return margin + 1e-30f;   // (products below the smallest normal number round absolutely)
    }
};

// One CTA per query: the kcand best of its row of `n` nominating scores, re-scored in the reference's operation
// order (an FMA chain over the dimensions, one thread per candidate: FP32Quantizer::ComputeDistImpl,
// src/quantization/fp32_quantizer.cpp:163-190; HalfPrecisionQuantizer,
// src/quantization/scalar_quantization/half_precision_quantizer.cpp:54-123), the k best of those as results.
// Infinite scores belong to rows that are filtered out.  A query is sure of its results when the k-th of them is nearer
// than the last nominated score allows any other row to be; the others are listed for an exact pass (bf_stream_kernel).
// Without the test a data offset of 50 (128 dimensions, spread 0.1) left a fifth of the true neighbours among the nominated.
template <typename E, int T>
__global__ void __launch_bounds__(T)
bf_rows_kernel(const float* __restrict__ scores, uint64_t ld, uint32_t n, const E* __restrict__ queries, uint32_t dim,
               const E* __restrict__ base, uint32_t kcand, uint32_t k, int metric, const int64_t* __restrict__ labels,
               int64_t* __restrict__ ids, float* __restrict__ dists, const BfMargin m) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SelectScratch sel;
    __shared__ __align__(16) uint64_t keys[SELECT_CAP];
    __shared__ __align__(16) uint64_t best[1024];
    __shared__ float s_qq, s_top;
    float* qf = reinterpret_cast<float*>(smem);
    const uint64_t q = blockIdx.x;
    for (uint32_t d = threadIdx.x; d < dim; d += T) {
        qf[d] = widen(queries[q * dim + d]);
    }
    const ScoreSource<true> src{reinterpret_cast<const uint32_t*>(scores + q * ld)};
    uint32_t left;   // no score that was not collected is below it
    const uint32_t have = block_select<T>(src, [](uint32_t i) { return i; }, n, kcand, keys, sel, &left);
    const bool dropped = left < ORDERED_INF;
    const float last = dropped ? ordered_to_float(left) : 0.f;
    if (threadIdx.x / 32 == T / 32 - 1) {   // (while the first warps wait for the candidates' rows)
        const float top = __ldg(m.row_max);
        float qq = 0.f;
        for (uint32_t d = threadIdx.x % 32; d < dim; d += 32) {
            qq = fmaf(qf[d], qf[d], qq);
        }
        for (int o = 16; o > 0; o >>= 1) {
            qq += __shfl_xor_sync(0xffffffffu, qq, o);
        }
        s_qq = qq;
        s_top = top;
    }
    for (uint32_t i = threadIdx.x; i < have; i += T) {
        const uint32_t row = static_cast<uint32_t>(keys[i]);
        keys[i] = make_key(row_exact_distance(base + static_cast<uint64_t>(row) * dim, qf, dim, metric == VB200_METRIC_L2), row);
    }
    block_sort_to<T>(keys, have, k, best);
    for (uint32_t i = threadIdx.x; i < k; i += T) {
        const bool there = i < have;
        ids[q * k + i] = there ? __ldg(labels + static_cast<uint32_t>(best[i])) : -1;
        dists[q * k + i] = there ? ordered_to_float(static_cast<uint32_t>(best[i] >> 32)) : INFINITY;
    }
    if (threadIdx.x == 0) {
        const bool l2 = metric == VB200_METRIC_L2;
        const float kth = dropped ? ordered_to_float(static_cast<uint32_t>(best[k - 1] >> 32)) : 0.f;
        const float qq = s_qq, margin = m.of(l2, s_top, qq, kth);
        // not finite: scores may have overflowed, and rows with them are not even among the counted
        if (!(margin < INFINITY) || (dropped && !(kth < last + (l2 ? qq : 1.0f) - margin))) {
            m.unsure[1 + atomicAdd(m.unsure, 1u)] = m.q_base + static_cast<uint32_t>(q);
        }
    }
}

// thr[q] = the next float above the kcand-th smallest of the query's n minima (+inf with fewer numbers among them), and
// spilled[q] = 0.  A CTA per query.
constexpr int BF_THRESHOLD_THREADS = 128;

__global__ void __launch_bounds__(BF_THRESHOLD_THREADS)
bf_threshold_kernel(const float* __restrict__ minima, uint32_t n, uint32_t kcand, float* __restrict__ thr, uint32_t* __restrict__ spilled) {
    __shared__ SelectScratch sel;
    const float* mine = minima + static_cast<uint64_t>(blockIdx.x) * n;
    uint32_t upto;
    const uint32_t bound = block_bound<BF_THRESHOLD_THREADS>(load_source([&](uint32_t i) { return float_to_ordered(__ldg(mine + i)); }), n, kcand,
                                                             kcand + kcand / 8 + 8, sel, &upto);
    if (threadIdx.x == 0) {
        thr[blockIdx.x] = bound >= ORDERED_INF ? INFINITY : ordered_to_float(bound + 1);
        spilled[blockIdx.x] = 0;
    }
}

// The rows that score below a query's threshold, as tc_collect left them, to the query's results.
struct BfCollected {
    const uint64_t* keys;     // [queries][lists][cap] nominating score and row
    const uint32_t* count;    // [queries][lists] entries offered; those past `cap` are in the spill
    const uint64_t* spill;    // [queries][room]
    const uint32_t* spilled;  // [queries] entries offered to it
    const float* thr;         // [queries]
    uint32_t lists, cap;
    uint32_t room;            // entries of one query that shared memory holds
    const void* queries;      // [queries x dim] in the index's type
    const void* base;
    uint32_t dim, kcand, k;
    int metric;
    const int64_t* labels;
    int64_t* ids;
    float* dists;
    BfMargin m;
};

// One CTA per query: gathers its lists, re-scores the kcand best in the reference's operation order (see bf_rows_kernel) and
// keeps k.  A query is sure of its results when the k-th of them is nearer than the last nominated score -- or the threshold, if
// no row below it was left out -- allows any other row to be.  When it is not, all collected rows are re-scored, after which
// only those above the threshold are left out; what is not sure then, or did not fit, is listed for the exact pass.
// Dynamic shared memory: [room] keys, [lists + 2] places, the query.
template <typename E, int T>
__global__ void __launch_bounds__(T)
bf_collected_kernel(const BfCollected p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SelectScratch sel;
    __shared__ __align__(16) uint64_t keys[SELECT_CAP];
    __shared__ __align__(16) uint64_t best[1024];
    __shared__ float s_qq, s_top;
    uint64_t* all = reinterpret_cast<uint64_t*>(smem);
    uint32_t* place = reinterpret_cast<uint32_t*>(all + p.room);
    float* qf = reinterpret_cast<float*>(place + p.lists + 2);
    const uint64_t q = blockIdx.x;
    const uint32_t dim = p.dim;
    const bool l2 = p.metric == VB200_METRIC_L2;
    const E* base = static_cast<const E*>(p.base);
    for (uint32_t d = threadIdx.x; d < dim; d += T) {
        qf[d] = widen(static_cast<const E*>(p.queries)[q * dim + d]);
    }
    __syncthreads();
    // where each list's entries begin, the spill's as the last of them
    const uint32_t* count = p.count + q * p.lists;
    uint32_t total = 0;
    for (uint32_t l0 = 0; l0 <= p.lists; l0 += T) {
        const uint32_t l = l0 + threadIdx.x;
        const uint32_t c = l < p.lists ? min(__ldg(count + l), p.cap) : (l == p.lists ? __ldg(p.spilled + q) : 0u);
        const uint32_t incl = block_inclusive_sum<T>(c, sel.warp_part);
        if (l <= p.lists) {
            place[l] = total + incl - c;
        }
        if (threadIdx.x == T - 1) {
            sel.total = total + incl;
        }
        __syncthreads();
        total = sel.total;
    }
    if (threadIdx.x == 0) {
        place[p.lists + 1] = total;
    }
    __syncthreads();
    if (total > p.room) {   // (so a spill that is not whole is not read)
        if (threadIdx.x == 0) {
            p.m.unsure[1 + atomicAdd(p.m.unsure, 1u)] = p.m.q_base + static_cast<uint32_t>(q);
        }
        return;
    }
    const uint64_t* mine = p.keys + q * p.lists * p.cap;
    for (uint32_t i = threadIdx.x; i < total; i += T) {
        uint32_t lo = 0, hi = p.lists + 1;   // the list that holds entry i is the last one that begins at or before it
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (place[mid] <= i) {
                lo = mid;
            } else {
                hi = mid;
            }
        }
        all[i] = __ldg((lo < p.lists ? mine + static_cast<uint64_t>(lo) * p.cap : p.spill + q * p.room) + (i - place[lo]));
    }
    __syncthreads();
    // a few more than the `keep` smallest of `all`, unsorted, in keys; how many.  No other is below *left (ORDERED_INF: no other)
    auto smallest = [&](uint32_t keep, uint32_t* left) -> uint32_t {
        return block_select<T>(load_source([&](uint32_t i) { return static_cast<uint32_t>(all[i] >> 32); }),
                               [&](uint32_t i) { return static_cast<uint32_t>(all[i]); }, total, keep, keys, sel, left);
    };
    uint32_t left;
    uint32_t have = smallest(p.kcand, &left);
    const float thr = __ldg(p.thr + q);
    float last = left < ORDERED_INF ? ordered_to_float(left) : thr;
    bool dropped = last < INFINITY;
    if (threadIdx.x / 32 == T / 32 - 1) {   // (while the first warps wait for the candidates' rows)
        const float top = __ldg(p.m.row_max);
        float qq = 0.f;
        for (uint32_t d = threadIdx.x % 32; d < dim; d += 32) {
            qq = fmaf(qf[d], qf[d], qq);
        }
        for (int o = 16; o > 0; o >>= 1) {
            qq += __shfl_xor_sync(0xffffffffu, qq, o);
        }
        s_qq = qq;
        s_top = top;
    }
    for (uint32_t i = threadIdx.x; i < have; i += T) {
        const uint32_t row = static_cast<uint32_t>(keys[i]);
        keys[i] = make_key(row_exact_distance(base + static_cast<uint64_t>(row) * dim, qf, dim, l2), row);
    }
    block_sort_to<T>(keys, have, p.k, best);
    const float top = s_top, qq = s_qq;
    auto sure = [&]() -> bool {
        if (dropped && have < p.k) {
            return false;
        }
        const float kth = dropped ? ordered_to_float(static_cast<uint32_t>(best[p.k - 1] >> 32)) : 0.f;
        const float margin = p.m.of(l2, top, qq, kth);
        return margin < INFINITY && (!dropped || kth < last + (l2 ? qq : 1.0f) - margin);
    };
    bool done = sure();
    if (!done && have < total) {
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < total; i += T) {
            const uint32_t row = static_cast<uint32_t>(all[i]);
            all[i] = make_key(row_exact_distance(base + static_cast<uint64_t>(row) * dim, qf, dim, l2), row);
        }
        __syncthreads();
        have = smallest(p.k, &left);
        block_sort_to<T>(keys, have, p.k, best);
        last = thr;
        dropped = thr < INFINITY;
        done = sure();
    }
    for (uint32_t i = threadIdx.x; i < p.k; i += T) {
        const bool there = i < have;
        p.ids[q * p.k + i] = there ? __ldg(p.labels + static_cast<uint32_t>(best[i])) : -1;
        p.dists[q * p.k + i] = there ? ordered_to_float(static_cast<uint32_t>(best[i] >> 32)) : INFINITY;
    }
    if (!done && threadIdx.x == 0) {
        p.m.unsure[1 + atomicAdd(p.m.unsure, 1u)] = p.m.q_base + static_cast<uint32_t>(q);
    }
}

}  // namespace vb200
