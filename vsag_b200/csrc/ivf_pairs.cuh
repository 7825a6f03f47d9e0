// Searches of small batches: every (query, probed list) pair is scanned on its own.
//
// When a list is probed by only a few queries of the batch there is nothing to gain from collecting the queries
// of a list into a tile, and the passes that do it (count, prefix sums, work items, places), the bounds and the
// second phase cost more than the rows.  Such a batch takes three or four launches here instead of fifteen:
//   row_chains_kernel     every centroid distance, as the reference's chain (no candidates, no re-scoring)
//   pairs_prepare_kernel  a CTA per query: its nprobe nearest lists, where each list's scores go, SQ8 weights
//   pair_scan_kernel      a CTA per (pair, 128 rows): one score per row, written where the CTA above said
//   scan_finalize_kernel  a CTA per query: the k best of its scores, exact re-scoring, rerank, labels
#pragma once

#include <cuda_bf16.h>

#include "block_select.cuh"
#include "row_scan.cuh"

namespace vb200 {

constexpr int PAIR_THREADS = 256;   // of the per-query kernels

struct PairTable {
    uint32_t* base;    // [nq x nprobe] a pair's first score within its query's stretch
    uint32_t* rows;    // [nq] scores of each query
    uint64_t stride;   // scores between the stretches of neighbouring queries
    float* scores;
    // Tiles: every pair starts on a multiple of 32 scores (rows past a list's end count as filtered) and the smallest
    // of each 32 stands, as an ordered value, in minima[query * stride / 32 + place / 32].  null: pairs back to back.
    uint32_t* minima;
};

// out[(q, r)] for every row r of `rows` and query q: L2 = sum of fma(t, t, .), t = row - query; otherwise the
// inner product chain, as it is (ONE_MINUS 0) or taken from one (1).  Every chain is one thread's, over ascending dimensions.
//
// A tile of 8 TM queries x 16 TN rows per CTA, TM x TN chains a thread, both operands CHAIN_K dimensions at a time through shared
// memory, CHAIN_STAGES deep.  Bound by the FMA pipe where there are CTAs for all SMs (4 x 4 chains: eight 16-byte reads of shared
// memory per 64 steps); 2 x 2 chains where that leaves SMs without one, whose time is the chain's latency.  1000 x 960 outputs of
// 960 dimensions: 197 us as a thread per row with eight queries (nine reads for 32 steps, two CTAs an SM), 77 now; 100 x 1024 of
// 640: 27.5, 17 now.
constexpr int CHAIN_THREADS = 128;
constexpr uint32_t CHAIN_K = 32;
constexpr int CHAIN_STAGES = 4;
constexpr uint32_t CHAIN_PITCH = CHAIN_K + 4;   // floats between rows in shared memory: 16-byte reads of neighbouring rows meet no bank twice

template <bool L2, int TM, int TN, int UNIT>
__global__ void __launch_bounds__(CHAIN_THREADS)
row_chains_kernel(const float* __restrict__ queries, uint32_t nq, uint64_t q_stride, const float* __restrict__ rows, uint32_t n_rows,
                  uint32_t dim, int one_minus, float* __restrict__ out, uint64_t ld) {
    constexpr uint32_t M = 8 * TM, N = 16 * TN, ELEMS = UNIT / 4;
    extern __shared__ __align__(16) unsigned char smem[];
    float* const stages = reinterpret_cast<float*>(smem);
    const uint32_t tx = threadIdx.x & 15u, ty = threadIdx.x >> 4;
    const uint32_t n0 = blockIdx.x * N, q0 = blockIdx.y * M;
    const uint32_t steps = (dim + CHAIN_K - 1) / CHAIN_K;
    auto request = [&](uint32_t step) {
        if (step < steps) {
            float* to = stages + step % CHAIN_STAGES * (M + N) * CHAIN_PITCH;
            constexpr uint32_t PER_ROW = CHAIN_K / ELEMS;
            for (uint32_t u = threadIdx.x; u < (M + N) * PER_ROW; u += CHAIN_THREADS) {
                const uint32_t r = u / PER_ROW, k = u % PER_ROW * ELEMS, d = step * CHAIN_K + k;
                const bool query = r < M;
                const uint32_t at = query ? q0 + r : n0 + r - M;
                const bool there = d < dim && at < (query ? nq : n_rows);
                // (what is not there is zero: a step of it adds nothing to a chain)
                const float* from = query ? queries + (there ? at * q_stride + d : 0) : rows + (there ? static_cast<uint64_t>(at) * dim + d : 0);
                const uint32_t bytes = there ? UNIT : 0;
                if (UNIT == 16) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(to + r * CHAIN_PITCH + k)), "l"(from), "r"(bytes)
                                 : "memory");
                } else {
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_u32(to + r * CHAIN_PITCH + k)), "l"(from), "r"(bytes)
                                 : "memory");
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < CHAIN_STAGES - 1; ++s) {
        request(s);
    }
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i) {
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            acc[i][j] = 0.f;
        }
    }
    auto chain = [](float& a, float x, float q) {
        if (L2) {
            const float t = __fsub_rn(x, q);
            a = fmaf(t, t, a);
        } else {
            a = fmaf(x, q, a);
        }
    };
    for (uint32_t step = 0; step < steps; ++step) {
        cp_async_wait_group<CHAIN_STAGES - 2>();
        __syncthreads();   // this step's operands are here for everybody, and nobody reads the step before any more
        request(step + CHAIN_STAGES - 1);
        const float* a_at = stages + step % CHAIN_STAGES * (M + N) * CHAIN_PITCH;
        const float* b_at = a_at + M * CHAIN_PITCH;
#pragma unroll
        for (uint32_t k = 0; k < CHAIN_K; k += 4) {
            float4 a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                a[i] = *reinterpret_cast<const float4*>(a_at + (ty + 8 * i) * CHAIN_PITCH + k);
            }
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                b[j] = *reinterpret_cast<const float4*>(b_at + (tx + 16 * j) * CHAIN_PITCH + k);
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    chain(acc[i][j], b[j].x, a[i].x);
                    chain(acc[i][j], b[j].y, a[i].y);
                    chain(acc[i][j], b[j].z, a[i].z);
                    chain(acc[i][j], b[j].w, a[i].w);
                }
            }
        }
    }
    cp_async_wait_group<0>();
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const uint32_t q = q0 + ty + 8 * i;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const uint32_t row = n0 + tx + 16 * j;
            if (q < nq && row < n_rows) {
                out[q * ld + row] = (!L2 && one_minus != 0) ? __fsub_rn(1.0f, acc[i][j]) : acc[i][j];
            }
        }
    }
}

struct PairsPrepare {
    const float* dist;        // [nq x ld] exact centroid distances, or
    const float* scores;      // [nq x ld] scores that nominate ncand centroids for exact distances; both null: `probes` is given
    uint64_t ld;
    uint32_t nlist, nprobe, ncand;
    const float* centroids;   // [nlist x dim] (with scores)
    int32_t* probes;          // [nq x nprobe] nearest first
    float* probe_dists;       // [nq x nprobe] or null
    const uint32_t* list_off;
    PairTable t;
    uint32_t* repeats;        // probes that a caller gave may name a list twice, which a query's stretch of scores has no room
                              // for: the later one is taken out and *repeats becomes 1; null: the probes are distinct
    uint32_t* count;          // [nlist] += 1 per pair of a list that is not empty, or null
    uint32_t* rank;           // [nq x nprobe] which of its list's pairs each is (0xFFFFFFFF: empty list)
    // SQ8 (null qw8: none): the int8 weight terms, their scale and the query's constant (see sq8_query_prep_kernel)
    const float* queries;
    uint32_t dim, dpad;
    const float *scale, *mid;
    int metric;
    int8_t* qw8;              // [nq][3][qstride]
    uint32_t qstride;
    float *qscale, *qa;
    // fp32 / bf16 / fp16 tiles (null: none): the query as operand rows of the tile scan, [nq][2 or 1][term_dims] 16-bit
    uint16_t* terms;
    uint32_t term_dims;       // a multiple of 64, zero past dim
    int term_fmt;             // ROW_F32, ROW_F32_SPLIT: bf16 hi and lo terms, ROW_BF16 / ROW_FP16: the codes
    __host__ __device__ uint32_t
    term_count() const {
        return term_fmt == ROW_F32 || term_fmt == ROW_F32_SPLIT ? 2 : 1;
    }
    // The same for the queries from q0 on (dist and scores are the caller's to set).
    PairsPrepare
    from(uint64_t q0) const {
        PairsPrepare p = *this;
        p.probes += q0 * nprobe;
        p.probe_dists += p.probe_dists != nullptr ? q0 * nprobe : 0;
        p.queries += q0 * dim;
        if (p.t.rows != nullptr) {
            p.t.base += q0 * nprobe;
            p.t.rows += q0;
        }
        if (p.count != nullptr) {
            p.rank += q0 * nprobe;
        }
        if (p.qw8 != nullptr) {
            p.qw8 += q0 * 3 * qstride;
            p.qscale += q0;
            p.qa += q0;
        }
        if (p.terms != nullptr) {
            p.terms += q0 * term_dims * term_count();
        }
        return p;
    }
};

__device__ __forceinline__ float
pair_block_sum(float v, float* part) {
    for (int o = 16; o > 0; o >>= 1) {
        v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        part[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    v = 0.f;
    for (int w = 0; w < PAIR_THREADS / 32; ++w) {
        v += part[w];
    }
    return v;
}

__device__ __forceinline__ float
pair_block_max(float v, float* part) {
    for (int o = 16; o > 0; o >>= 1) {
        v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        part[threadIdx.x >> 5] = v;
    }
    __syncthreads();
    v = part[0];
    for (int w = 1; w < PAIR_THREADS / 32; ++w) {
        v = fmaxf(v, part[w]);
    }
    return v;
}

// The query as operand rows of the tile scan, by `threads` threads.
__device__ __forceinline__ void
pair_query_terms(const PairsPrepare& p, uint64_t q, const float* src, uint32_t thread, uint32_t threads) {
    uint16_t* t = p.terms + q * p.term_dims * p.term_count();
    for (uint32_t e = thread; e < p.term_dims; e += threads) {
        if (p.term_count() == 2) {
            // converted rows: place e of a piece of 64, unit e / 8, holds dimensions 4 u .. + 3 and 32 + 4 u .. + 3 (tile_scan_kernel)
            const uint32_t u = (e & 63u) >> 3, i = e & 7u;
            const uint32_t d = p.term_fmt == ROW_F32_SPLIT ? e : (e & ~63u) + (i < 4 ? 4 * u + i : 28 + 4 * u + i);
            const float v = d < p.dim ? __ldg(src + d) : 0.f;
            const __nv_bfloat16 hi = __float2bfloat16_rn(v);
            t[e] = __bfloat16_as_ushort(hi);
            t[p.term_dims + e] = __bfloat16_as_ushort(__float2bfloat16_rn(v - __bfloat162float(hi)));
        } else if (e >= p.dim) {
            t[e] = 0;
        } else {
            t[e] = p.term_fmt == ROW_BF16 ? half_encode<SCAN_FMT_BF16>(__ldg(src + e)) : half_encode<SCAN_FMT_FP16>(__ldg(src + e));
        }
    }
}

// The int8 terms of a query's SQ8 weights, s = their scale.
__device__ __forceinline__ void
pair_query_weights(const PairsPrepare& p, uint64_t q, const float* src, float s, uint32_t thread, uint32_t threads) {
    int8_t* t = p.qw8 + q * 3 * p.qstride;
    for (uint32_t d = thread; d < p.qstride; d += threads) {
        const float u = d < p.dim ? __ldg(src + d) * __ldg(p.scale + d) / s : 0.f;
        const float t1 = fminf(fmaxf(rintf(u), -127.f), 127.f);
        const float v2 = (u - t1) * 254.0f;
        const float t2 = fminf(fmaxf(rintf(v2), -127.f), 127.f);
        const float t3 = fminf(fmaxf(rintf((v2 - t2) * 254.0f), -127.f), 127.f);
        t[d] = static_cast<int8_t>(static_cast<int>(t1));
        t[p.qstride + d] = static_cast<int8_t>(static_cast<int>(t2));
        t[2 * p.qstride + d] = static_cast<int8_t>(static_cast<int>(t3));
    }
}

__global__ void __launch_bounds__(PAIR_THREADS)
pairs_prepare_kernel(const PairsPrepare p) {
    __shared__ SelectScratch sel;
    __shared__ __align__(16) uint64_t keys[SELECT_CAP];
    __shared__ __align__(16) uint64_t best[1024];
    __shared__ float part[PAIR_THREADS / 32];
    const uint64_t q = blockIdx.x;
    int32_t* probes = p.probes + q * p.nprobe;
    if (p.dist != nullptr || p.scores != nullptr) {
        uint32_t found;
        if (p.scores != nullptr) {
            // IVF::route_buckets_only's loop (src/algorithm/ivf/ivf.cpp:1589-1660) over the nominated centroids:
            // distance ascending, lower list id first on ties
            extern __shared__ __align__(16) unsigned char smem[];
            float* qs = reinterpret_cast<float*>(smem);
            for (uint32_t d = threadIdx.x; d < p.dim; d += PAIR_THREADS) {
                qs[d] = __ldg(p.queries + q * p.dim + d);
            }
            const ScoreSource<> src{reinterpret_cast<const uint32_t*>(p.scores + q * p.ld)};
            // (what was collected, usually a few more than ncand, is scored as it is: ordering it first cost more)
            found = block_select<PAIR_THREADS>(src, [](uint32_t i) { return i; }, p.nlist, p.ncand, keys, sel);
            for (uint32_t i = threadIdx.x; i < found; i += PAIR_THREADS) {
                const uint32_t l = static_cast<uint32_t>(keys[i]);
                keys[i] = make_key(row_exact_distance(p.centroids + static_cast<uint64_t>(l) * p.dim, qs, p.dim, p.metric == VB200_METRIC_L2), l);
            }
        } else {
            const float* row = p.dist + q * p.ld;
            found = block_select<PAIR_THREADS>(load_source([&](uint32_t i) { return float_to_ordered(__ldg(row + i)); }),
                                               [](uint32_t i) { return i; }, p.nlist, p.nprobe, keys, sel);
        }
        block_sort_to<PAIR_THREADS>(keys, found, p.nprobe, best);
        for (uint32_t i = threadIdx.x; i < p.nprobe; i += PAIR_THREADS) {
            const bool have = i < found;
            probes[i] = have ? static_cast<int32_t>(static_cast<uint32_t>(best[i])) : -1;
            if (p.probe_dists != nullptr) {
                p.probe_dists[q * p.nprobe + i] = have ? ordered_to_float(static_cast<uint32_t>(best[i] >> 32)) : INFINITY;
            }
        }
        __syncthreads();
    }
    if (p.t.rows == nullptr) {
        return;   // only the routing is wanted
    }
    const uint32_t round = p.t.minima != nullptr ? 31u : 0u;
    uint32_t run = 0;
    for (uint32_t i0 = 0; i0 < p.nprobe; i0 += PAIR_THREADS) {
        const uint32_t i = i0 + threadIdx.x;
        uint32_t len = 0;
        if (i < p.nprobe) {
            int32_t l = probes[i];
            if (p.repeats != nullptr && l >= 0) {
                // (the first of its kind is never changed, so it does not matter which of the others is gone already)
                bool again = false;
                for (uint32_t j = 0; j < i && !again; ++j) {
                    again = *const_cast<const volatile int32_t*>(probes + j) == l;
                }
                if (again) {
                    l = probes[i] = -1;
                    *p.repeats = 1;
                }
            }
            if (l >= 0 && static_cast<uint32_t>(l) < p.nlist) {
                len = p.list_off[l + 1] - p.list_off[l];
            }
            if (p.count != nullptr) {
                p.rank[q * p.nprobe + i] = len > 0 ? atomicAdd(p.count + l, 1u) : 0xFFFFFFFFu;
            }
            len = (len + round) & ~round;
        }
        const uint32_t incl = block_inclusive_sum<PAIR_THREADS>(len, sel.warp_part);
        if (i < p.nprobe) {
            p.t.base[q * p.nprobe + i] = run + incl - len;
        }
        if (threadIdx.x == PAIR_THREADS - 1) {
            sel.total = run + incl;
        }
        __syncthreads();
        run = sel.total;
    }
    if (threadIdx.x == 0) {
        p.t.rows[q] = run;
    }
    const float* src = p.queries + q * p.dim;
    if (p.terms != nullptr) {
        pair_query_terms(p, q, src, threadIdx.x, PAIR_THREADS);
    }
    if (p.qw8 == nullptr) {
        return;
    }
    float qq = 0.f, qm = 0.f, wmax = 0.f;
    for (uint32_t d = threadIdx.x; d < p.dim; d += PAIR_THREADS) {
        const float v = __ldg(src + d);
        qq = fmaf(v, v, qq);
        qm = fmaf(v, __ldg(p.mid + d), qm);
        wmax = fmaxf(wmax, fabsf(v * __ldg(p.scale + d)));
    }
    qq = pair_block_sum(qq, part);
    qm = pair_block_sum(qm, part);
    wmax = pair_block_max(wmax, part);
    const float s = wmax > 0.f && wmax < INFINITY ? wmax / 127.0f : 1.0f;
    pair_query_weights(p, q, src, s, threadIdx.x, PAIR_THREADS);
    if (threadIdx.x == 0) {
        p.qscale[q] = s;
        p.qa[q] = p.metric == VB200_METRIC_L2 ? fmaf(-2.0f, qm, qq) : 1.0f - qm;
    }
}

// pairs_prepare_kernel with a warp per query, for routing that selects WARP_SELECT_MAX lists or candidates at most and lists that are
// distinct (p.repeats null): no barriers.  1000 queries against 1024 lists, 40 candidates: 32 us with a CTA per query, 20 this way; 4096 lists,
// 72 candidates of 960 dimensions: 122, 97.
// Dynamic shared memory per warp: [WARP_SELECT_CAP] keys, and the stages of warp_rows and the query where candidates are re-scored.
constexpr int PREPARE_WARPS = 2;
constexpr int PREPARE_SUMS = PAIR_THREADS / 32;   // partial sums of a lane: 256 of a query, as a CTA's threads have them (scan_finalize_kernel's margin)

__host__ __device__ inline size_t
prepare_warp_bytes(bool rescore, uint32_t dim) {
    return WARP_SELECT_CAP * sizeof(uint64_t) + (rescore ? WARP_ROWS_BYTES + (static_cast<size_t>(dim) + 3) / 4 * 16 : 0);
}

// The exact distances of the centroids named by the low words of keys[0 .. count), as keys (one warp).
__device__ __forceinline__ void
warp_centroid_distances(const float* centroids, uint32_t dim, bool l2, const float* qs, uint32_t count, uint64_t* keys, unsigned char* stages,
                        uint32_t lane) {
    if (dim % 4 != 0 || (reinterpret_cast<uintptr_t>(centroids) & 15u) != 0) {   // rows that are not 16-byte aligned
        for (uint32_t i = lane; i < count; i += 32) {
            const uint32_t l = static_cast<uint32_t>(keys[i]);
            keys[i] = make_key(row_exact_distance(centroids + static_cast<uint64_t>(l) * dim, qs, dim, l2), l);
        }
        __syncwarp();
        return;
    }
    const auto row = [&](uint32_t i) { return reinterpret_cast<const unsigned char*>(centroids + static_cast<uint64_t>(static_cast<uint32_t>(keys[i])) * dim); };
    // (a key is replaced when its batch of rows is done and its row has been read)
    if (l2) {
        RowAcc<ROW_F32, true, 1> acc;
        warp_rows(count, row, dim * 4, dim, qs, 0, stages, lane, acc,
                  [&](uint32_t i, const auto& a) { keys[i] = make_key(a.acc[0], static_cast<uint32_t>(keys[i])); });
    } else {
        RowAcc<ROW_F32, false, 1> acc;
        warp_rows(count, row, dim * 4, dim, qs, 0, stages, lane, acc,
                  [&](uint32_t i, const auto& a) { keys[i] = make_key(__fsub_rn(1.0f, a.acc[0]), static_cast<uint32_t>(keys[i])); });
    }
}

__global__ void __launch_bounds__(PREPARE_WARPS * 32)
pairs_prepare_warps_kernel(const PairsPrepare p, uint64_t nq) {
    extern __shared__ __align__(16) unsigned char smem[];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t q = static_cast<uint64_t>(blockIdx.x) * PREPARE_WARPS + warp;
    if (q >= nq) {
        return;
    }
    unsigned char* mine = smem + warp * prepare_warp_bytes(p.scores != nullptr, p.dim);
    uint64_t* keys = reinterpret_cast<uint64_t*>(mine);
    int32_t* probes = p.probes + q * p.nprobe;
    const float* query = p.queries + q * p.dim;
    if (p.dist != nullptr || p.scores != nullptr) {
        const float* row = (p.scores != nullptr ? p.scores : p.dist) + q * p.ld;
        const uint32_t wanted = p.scores != nullptr ? p.ncand : p.nprobe;
        const auto load = [&](uint32_t i) { return float_to_ordered(__ldg(row + i)); };
        const auto number = [](uint32_t i) { return i; };
        uint32_t left;
        uint32_t found = warp_select(load, number, p.nlist, wanted, keys, lane, &left);
        if (found > WARP_SELECT_CAP) {
            // Many at the bound.  The smallest value that `wanted` are at or below, then of those equal to it the first ones.
            uint32_t low = 0, high = left;
            while (low < high) {
                const uint32_t mid = low + (high - low) / 2;
                uint32_t count = 0;
                warp_walk(load, p.nlist, lane, [&](uint32_t, uint32_t u, uint32_t) { count += u <= mid ? 1u : 0u; });
                count = __reduce_add_sync(0xffffffffu, count);
                if (count < wanted) {
                    low = mid + 1;
                } else {
                    high = mid;
                }
            }
            found = high > 0 ? warp_collect(load, number, p.nlist, high - 1, keys, lane) : 0u;
            warp_walk(load, p.nlist, lane, [&](uint32_t i, uint32_t u, uint32_t) {
                const uint32_t mask = __ballot_sync(0xffffffffu, u == high && u <= ORDERED_INF);
                const uint32_t at = found + __popc(mask & ((1u << lane) - 1u));
                if (u == high && u <= ORDERED_INF && at < wanted) {
                    keys[at] = (static_cast<uint64_t>(u) << 32) | i;
                }
                found = min(found + __popc(mask), wanted);
            });
            __syncwarp();
        }
        if (p.scores != nullptr) {
            // IVF::route_buckets_only's loop (src/algorithm/ivf/ivf.cpp:1589-1660) over the nominated centroids:
            // distance ascending, lower list id first on ties
            unsigned char* stages = reinterpret_cast<unsigned char*>(keys + WARP_SELECT_CAP);
            float* qs = reinterpret_cast<float*>(stages + WARP_ROWS_BYTES);
            for (uint32_t d = lane; d < p.dim; d += 32) {
                qs[d] = __ldg(query + d);
            }
            __syncwarp();
            warp_centroid_distances(p.centroids, p.dim, p.metric == VB200_METRIC_L2, qs, found, keys, stages, lane);
        }
        warp_sort(keys, found, lane);
        for (uint32_t i = lane; i < p.nprobe; i += 32) {
            const bool have = i < found;
            probes[i] = have ? static_cast<int32_t>(static_cast<uint32_t>(keys[i])) : -1;
            if (p.probe_dists != nullptr) {
                p.probe_dists[q * p.nprobe + i] = have ? ordered_to_float(static_cast<uint32_t>(keys[i] >> 32)) : INFINITY;
            }
        }
        __syncwarp();
    }
    if (p.t.rows == nullptr) {
        return;   // only the routing is wanted
    }
    const uint32_t round = p.t.minima != nullptr ? 31u : 0u;
    uint32_t run = 0;
    for (uint32_t i0 = 0; i0 < p.nprobe; i0 += 32) {
        const uint32_t i = i0 + lane;
        uint32_t len = 0;
        if (i < p.nprobe) {
            const int32_t l = probes[i];
            if (l >= 0 && static_cast<uint32_t>(l) < p.nlist) {
                len = __ldg(p.list_off + l + 1) - __ldg(p.list_off + l);
            }
            if (p.count != nullptr) {
                p.rank[q * p.nprobe + i] = len > 0 ? atomicAdd(p.count + l, 1u) : 0xFFFFFFFFu;
            }
            len = (len + round) & ~round;
        }
        uint32_t incl = len;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            incl += lane >= static_cast<uint32_t>(o) ? v : 0u;
        }
        if (i < p.nprobe) {
            p.t.base[q * p.nprobe + i] = run + incl - len;
        }
        run += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) {
        p.t.rows[q] = run;
    }
    if (p.terms != nullptr) {
        pair_query_terms(p, q, query, lane, 32);
    }
    if (p.qw8 == nullptr) {
        return;
    }
    float qq_part[PREPARE_SUMS] = {}, qm_part[PREPARE_SUMS] = {}, wmax = 0.f;
    for (uint32_t d0 = lane; d0 < p.dim; d0 += 32 * PREPARE_SUMS) {
#pragma unroll
        for (int j = 0; j < PREPARE_SUMS; ++j) {
            const uint32_t d = d0 + 32 * j;
            if (d < p.dim) {
                const float v = __ldg(query + d);
                qq_part[j] = fmaf(v, v, qq_part[j]);
                qm_part[j] = fmaf(v, __ldg(p.mid + d), qm_part[j]);
                wmax = fmaxf(wmax, fabsf(v * __ldg(p.scale + d)));
            }
        }
    }
#pragma unroll
    for (int w = PREPARE_SUMS / 2; w > 0; w /= 2) {
#pragma unroll
        for (int j = 0; j < w; ++j) {
            qq_part[j] += qq_part[j + w];
            qm_part[j] += qm_part[j + w];
        }
    }
    float qq = qq_part[0], qm = qm_part[0];
    for (int o = 16; o > 0; o >>= 1) {
        qq += __shfl_xor_sync(0xffffffffu, qq, o);
        qm += __shfl_xor_sync(0xffffffffu, qm, o);
        wmax = fmaxf(wmax, __shfl_xor_sync(0xffffffffu, wmax, o));
    }
    const float s = wmax > 0.f && wmax < INFINITY ? wmax / 127.0f : 1.0f;
    pair_query_weights(p, q, query, s, lane, 32);
    if (lane == 0) {
        p.qscale[q] = s;
        p.qa[q] = p.metric == VB200_METRIC_L2 ? fmaf(-2.0f, qm, qq) : 1.0f - qm;
    }
}

// RaBitQ queries: rotated rows t[nq x dim] -> the processed query (RaBitQuantizer::ProcessQueryImpl,
// rabitq_quantizer.cpp:2130-2217: centred, divided by the norm of the ascending chain, the norm behind) and, with
// qw8, the values sv_d = inv_sqrt_d * q_d of the estimator as three int8 terms, their scale and the terms' sums.  The
// chain is one thread's, over values the whole CTA put into shared memory.
__global__ void __launch_bounds__(PAIR_THREADS)
rabitq_query_kernel(const float* __restrict__ t, uint32_t dim, const float* __restrict__ centroid, uint32_t qstride, float inv_sqrt_d,
                    float* __restrict__ out, int8_t* __restrict__ qw8, float* __restrict__ qscale, int32_t* __restrict__ qsum) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ float part[PAIR_THREADS / 32];
    __shared__ float s_norm;
    __shared__ int32_t sums[3];
    float* df = reinterpret_cast<float*>(smem);
    const uint64_t q = blockIdx.x;
    const float* src = t + q * dim;
    for (uint32_t d = threadIdx.x; d < dim; d += PAIR_THREADS) {
        df[d] = __fsub_rn(__ldg(src + d), __ldg(centroid + d));
    }
    if (threadIdx.x < 3) {
        sums[threadIdx.x] = 0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
#pragma unroll 16
        for (uint32_t d = 0; d < dim; ++d) {
            s = fmaf(df[d], df[d], s);
        }
        s_norm = s < 1e-5f ? 1.0f : __fsqrt_rn(s);
        out[q * (dim + 1) + dim] = s_norm;
    }
    __syncthreads();
    const float norm = s_norm;
    float wmax = 0.f;
    for (uint32_t d = threadIdx.x; d < dim; d += PAIR_THREADS) {
        const float v = __fdiv_rn(df[d], norm);
        out[q * (dim + 1) + d] = v;
        const float w = __fmul_rn(inv_sqrt_d, v);
        df[d] = w;   // (this thread's own element)
        wmax = fmaxf(wmax, fabsf(w));
    }
    if (qw8 == nullptr) {
        return;
    }
    wmax = pair_block_max(wmax, part);
    const float s = wmax > 0.f && wmax < INFINITY ? wmax / 127.0f : 1.0f;
    int8_t* terms = qw8 + q * 3 * qstride;
    int32_t n1 = 0, n2 = 0, n3 = 0;
    for (uint32_t d = threadIdx.x; d < qstride; d += PAIR_THREADS) {
        const float u = d < dim ? df[d] / s : 0.f;
        const float t1 = fminf(fmaxf(rintf(u), -127.f), 127.f);
        const float v2 = (u - t1) * 254.0f;
        const float t2 = fminf(fmaxf(rintf(v2), -127.f), 127.f);
        const float t3 = fminf(fmaxf(rintf((v2 - t2) * 254.0f), -127.f), 127.f);
        // bit 8 b + s of 32 sign bits becomes byte 4 s + b of the tile scan's operand
        const uint32_t at = (d & ~31u) + (d & 7u) * 4 + ((d & 31u) >> 3);
        terms[at] = static_cast<int8_t>(static_cast<int>(t1));
        terms[qstride + at] = static_cast<int8_t>(static_cast<int>(t2));
        terms[2 * qstride + at] = static_cast<int8_t>(static_cast<int>(t3));
        n1 += static_cast<int>(t1);
        n2 += static_cast<int>(t2);
        n3 += static_cast<int>(t3);
    }
    n1 = __reduce_add_sync(0xffffffffu, n1);
    n2 = __reduce_add_sync(0xffffffffu, n2);
    n3 = __reduce_add_sync(0xffffffffu, n3);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sums[0], n1);
        atomicAdd(&sums[1], n2);
        atomicAdd(&sums[2], n3);
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        qsum[4 * q + threadIdx.x] = sums[threadIdx.x];
    }
    if (threadIdx.x == 0) {
        qscale[q] = s;
    }
}

// Squared norms of the stored rows and the largest norm (RaBitQ: |x|^2 and -2 |x| / error, largest norm / |error|;
// SQ8: of the norms already in `norm`).  A warp per row; top[] is cleared by the caller.
template <int FMT>
__global__ void __launch_bounds__(256)
record_norms_kernel(const uint8_t* __restrict__ codes, uint64_t n, uint32_t dim, uint32_t stride, float* __restrict__ norm,
                    float* __restrict__ top) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t warp = (static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x) >> 5, warps = static_cast<uint64_t>(gridDim.x) * 8;
    float most = 0.f, gain = 0.f;
    if (FMT == ROW_SQ8 || FMT == ROW_RABITQ) {
        for (uint64_t r = warp * 32 + lane; r < n; r += warps * 32) {
            if (FMT == ROW_SQ8) {
                most = fmaxf(most, norm[r]);
            } else {
                const float* tail = reinterpret_cast<const float*>(codes + r * stride + ((dim + 7) / 8 + 3) / 4 * 4);
                const float err = fabsf(tail[1]) < 1e-5f ? (tail[1] >= 0.f ? 1.0f : -1.0f) : tail[1];
                most = fmaxf(most, tail[0]);
                gain = fmaxf(gain, tail[0] / fabsf(err));
                reinterpret_cast<float2*>(norm)[r] = make_float2(tail[0] * tail[0], -2.0f * tail[0] / err);
            }
        }
    } else {
        for (uint64_t r = warp; r < n; r += warps) {
            float s = 0.f;
            for (uint32_t d = lane; d < dim; d += 32) {
                float v;
                if (FMT == ROW_F32) {
                    v = reinterpret_cast<const float*>(codes + r * stride)[d];
                } else {
                    v = half_decode<FMT == ROW_BF16 ? SCAN_FMT_BF16 : SCAN_FMT_FP16>(reinterpret_cast<const uint16_t*>(codes + r * stride)[d]);
                }
                s = fmaf(v, v, s);
            }
            for (int o = 16; o > 0; o >>= 1) {
                s += __shfl_xor_sync(0xffffffffu, s, o);
            }
            if (lane == 0) {
                norm[r] = s;
            }
            most = fmaxf(most, s);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, o));
        gain = fmaxf(gain, __shfl_xor_sync(0xffffffffu, gain, o));
    }
    if (lane == 0) {   // non-negative floats order like their bit patterns
        atomicMax(reinterpret_cast<int*>(top), __float_as_int(FMT == ROW_RABITQ ? most : sqrtf(most) * 1.000001f));
        atomicMax(reinterpret_cast<int*>(top + 1), __float_as_int(gain * 1.000001f));
    }
}

struct PairScan {
    ScanParams s;             // rows, list_off, filter, SQ8 / RaBitQ constants (queries = processed ones for RaBitQ)
    PairTable t;
    const int32_t* probes;
    uint32_t nprobe;
    uint32_t per_pair;        // CTAs per pair: CTA c takes chunks c, c + per_pair, ... of the list
    uint32_t row_bytes;       // of a row that the scan reads
    const int8_t* qw8;        // SQ8: [nq][3][dpad]
    const float* qscale;
    uint32_t qstride;         // query values in shared memory: floats (SQ8: bytes of a term)
};

// The bit pattern of the score of a row that the id filter rejects: a NaN, which no selection takes, and not the one that
// arithmetic results in (0x7FFFFFFF: a score that overflowed, whose exact distance may be finite).
constexpr uint32_t SCORE_FILTERED = 0x7FFFFFFEu;

// est, record norm and error -> the reference's distance (ivf_rabitq_scan_kernel).
__device__ __forceinline__ float
rabitq_distance(float ip, float bn, float err, float qn) {
    if (static_cast<double>(fabsf(err)) < 1e-5) {   // float compared with a double literal, as in the reference
        err = err >= 0.f ? 1.0f : -1.0f;
    }
    const float est = __fdiv_rn(ip, err);
    const float p3 = __fmul_rn(__fmul_rn(__fmul_rn(-2.0f, bn), qn), est);
    return __fadd_rn(__fadd_rn(__fmul_rn(bn, bn), __fmul_rn(qn, qn)), p3);
}

// The query of a pair as the codec's chain reads it, in shared memory (qstride values, zero padded).
template <int FMT>
__device__ __forceinline__ void
stage_query(const PairScan& p, uint64_t q, float* qs, uint32_t threads) {
    if (FMT == ROW_SQ8) {
        const uint4* src = reinterpret_cast<const uint4*>(p.qw8 + q * 3 * p.qstride);
        for (uint32_t i = threadIdx.x; i < 3 * p.qstride / 16; i += threads) {
            reinterpret_cast<uint4*>(qs)[i] = __ldg(src + i);
        }
        return;
    }
    const uint32_t dim = p.s.dim;
    const float* src = p.s.queries + q * (FMT == ROW_RABITQ ? dim + 1 : dim);
    for (uint32_t d = threadIdx.x; d < p.qstride; d += threads) {
        float v = d < dim ? __ldg(src + d) : 0.f;
        if (FMT == ROW_BF16) {
            v = half_decode<SCAN_FMT_BF16>(half_encode<SCAN_FMT_BF16>(v));
        } else if (FMT == ROW_FP16) {
            v = half_decode<SCAN_FMT_FP16>(half_encode<SCAN_FMT_FP16>(v));
        } else if (FMT == ROW_RABITQ) {
            v = __fmul_rn(p.s.inv_sqrt_d, v);
        }
        qs[d] = v;
    }
}

template <int FMT, bool L2>
__global__ void __launch_bounds__(RS_ROWS)
pair_scan_kernel(const PairScan p) {
    extern __shared__ __align__(16) unsigned char smem[];
    float* qs = reinterpret_cast<float*>(smem + RS_STAGES * RS_STAGE);
    const uint32_t pair = blockIdx.x / p.per_pair, first = blockIdx.x - pair * p.per_pair;
    const uint32_t q = pair / p.nprobe;
    const int32_t l = __ldg(p.probes + pair);
    if (l < 0 || static_cast<uint32_t>(l) >= p.s.nlist) {
        return;
    }
    const uint32_t lbeg = __ldg(p.s.list_off + l), len = __ldg(p.s.list_off + l + 1) - lbeg;
    if (first * RS_ROWS >= len) {
        return;
    }
    stage_query<FMT>(p, q, qs, RS_ROWS);
    uint32_t* out = reinterpret_cast<uint32_t*>(p.t.scores + q * p.t.stride + p.t.base[pair]);
    float qa = 0.f, cq = 0.f, qn = 0.f;
    if (FMT == ROW_SQ8) {
        qa = __ldg(p.s.qa + q);
        cq = p.s.coef_c * __ldg(p.qscale + q);
    } else if (FMT == ROW_RABITQ) {
        qn = __ldg(p.s.queries + static_cast<uint64_t>(q) * (p.s.dim + 1) + p.s.dim);
    }
    const uint8_t* rows = p.s.codes + static_cast<uint64_t>(lbeg) * p.s.code_stride;
    RowAcc<FMT, L2, 1> acc;
    row_stream<16>(rows, p.s.code_stride, p.row_bytes, p.s.dim, len, first, p.per_pair, smem, qs, p.qstride, acc,
                   [&](uint64_t row, bool valid) {
                       if (!valid) {
                           return;
                       }
                       const uint32_t pos = lbeg + static_cast<uint32_t>(row);
                       float v;
                       if constexpr (FMT == ROW_SQ8) {
                           const float f = sq8_term_sum(acc.a1[0], acc.a2[0], acc.a3[0], p.s.dim <= SQ8_NARROW_DIMS);
                           v = fmaf(cq, f, p.s.coef_b * __ldg(p.s.code_norm + pos)) + qa;
                       } else if constexpr (FMT == ROW_RABITQ) {
                           const float* tail = reinterpret_cast<const float*>(rows + row * p.s.code_stride + p.row_bytes);
                           v = rabitq_distance(acc.acc[0], __ldg(tail), __ldg(tail + 1), qn);
                       } else {
                           v = L2 ? acc.acc[0] : __fsub_rn(1.0f, acc.acc[0]);
                       }
                       uint32_t bits = __float_as_uint(v);
                       if (p.s.filter_pos_inner != nullptr && scan_row_filtered(p.s, pos)) {
                           bits = SCORE_FILTERED;
                       }
                       out[row] = bits;
                   });
}

struct ScanFinalize {
    PairScan scan;             // the scan whose scores are read
    uint32_t kscan, k;         // results of the scan per query; results of the search (fewer with a rerank)
    uint32_t kcand;            // candidates taken from the scores: kscan, and more when they are re-scored
    const float *lower, *diff; // SQ8
    const float* row_max;      // [0] largest row norm of the index; RaBitQ: [1] largest norm / |error|
    const float* queries;      // [nq x dim] plain queries (SQ8 re-scoring, rerank)
    const uint32_t* pos_inner;
    const int64_t* labels;
    uint32_t* rerank_ids;      // [nq x kscan] rerank: the candidates go here instead of to the results, or null
    uint32_t* rows_scanned;    // [nq] rows of each query's lists (pinned host memory)
    int64_t* ids;
    float* dists;
};

// Exact SQ8 distance in the reference's operation order (sq8_rescore_kernel); q, lower and diff in shared memory.
__device__ __forceinline__ float
sq8_exact_distance(const uint8_t* code, uint32_t dim, bool l2, const float* q, const float* lo, const float* di) {
    const float inv255 = 1.0f / 255.0f;
    float s = 0.f;
    for (uint32_t d0 = 0; d0 < dim; d0 += 64) {
        uint4 raw[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            raw[u] = d0 + u * 16 < dim ? __ldg(reinterpret_cast<const uint4*>(code + d0 + u * 16)) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t words[4] = {raw[u].x, raw[u].y, raw[u].z, raw[u].w};
#pragma unroll
            for (uint32_t j = 0; j < 16; ++j) {
                const uint32_t d = d0 + u * 16 + j;
                if (d < dim) {
                    const float byte = static_cast<float>((words[j >> 2] >> ((j & 3u) * 8)) & 0xFFu);
                    const float x = fmaf(__fmul_rn(byte, inv255), di[d], lo[d]);
                    if (l2) {
                        const float t = __fsub_rn(q[d], x);
                        s = fmaf(t, t, s);
                    } else {
                        s = fmaf(q[d], x, s);
                    }
                }
            }
        }
    }
    return l2 ? s : __fsub_rn(1.0f, s);
}

// A score's place among its query's -> the row's position: the pair whose stretch holds it is the last one that
// starts at or before the place (an empty list shares its start with the pair after it).
struct ScorePosition {
    const uint32_t* base;    // (shared memory) first place of every pair
    const uint32_t* start;   // (shared memory) first position of its list
    uint32_t nprobe;
    __device__ __forceinline__ uint32_t
    operator()(uint32_t i) const {
        uint32_t lo = 0, hi = nprobe;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) >> 1;
            if (base[mid] <= i) {
                lo = mid;
            } else {
                hi = mid;
            }
        }
        return start[lo] + (i - base[lo]);
    }
};

constexpr uint32_t FINAL_GROUPS = 1024;   // groups of 32 scores looked into at most

// Place number i of the scores in the listed groups -> the row's position.
struct GroupPosition {
    const uint32_t* ids;
    ScorePosition position;
    __device__ __forceinline__ uint32_t
    operator()(uint32_t i) const {
        return position(ids[i >> 5] * 32 + (i & 31u));
    }
};

// Exact distance of one code record in the reference's operation order; qc: the query as the codec's chain reads it
// (stage_query), zero padded.  Four 16-byte loads in flight.
template <int FMT, bool L2>
__device__ __forceinline__ float
record_exact_distance(const uint8_t* rec, uint32_t dim, uint32_t row_bytes, const float* qc, float qn) {
    RowAcc<FMT, L2, 1> acc;
    acc.clear();
    constexpr uint32_t UD = RowAcc<FMT, L2, 1>::UNIT_DIMS;
    const uint4* v = reinterpret_cast<const uint4*>(rec);
    const uint32_t units = (dim + UD - 1) / UD;
    for (uint32_t u0 = 0; u0 < units; u0 += 4) {
        uint4 w[4];
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            w[j] = u0 + j < units ? __ldg(v + u0 + j) : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t d0 = (u0 + j) * UD;
            if (d0 + UD <= dim) {
                acc.unit(w[j], qc, 0, d0);
            } else if (d0 < dim) {
                acc.tail(w[j], qc, 0, d0, dim - d0);
            }
        }
    }
    if constexpr (FMT == ROW_RABITQ) {
        const float* tail = reinterpret_cast<const float*>(rec + row_bytes);
        return rabitq_distance(acc.acc[0], __ldg(tail), __ldg(tail + 1), qn);
    } else {
        return L2 ? acc.acc[0] : __fsub_rn(1.0f, acc.acc[0]);
    }
}

// Dynamic shared memory: [2][nprobe] pair places and list starts; [SQ8] the plain query, lower and
// diff, or [other codecs re-scored after tiles] the query as the codec reads it (qstride floats).
// APPROX: the scores only rank (SQ8's integer form, tensor-core tiles).  The kcand best by score are re-scored
// exactly; a row that was not among them has an exact distance of at least (the last kept score - margin), margin
// bounding the difference between score and exact distance, so when the kscan-th exact distance is below that the
// result is the exact one.  Otherwise (scores crowded within the rounding of the arithmetic) every row of the query
// is scored exactly here.
// CTAS: CTAs an SM that the registers leave room for.  (Seven take 1000 queries together, 57 -> 41 us; the one-bit chain wants the
// registers, 244 -> 256, and so do few queries, for which nothing else hides the loads: 32 take 46 us, with seven 54.)
template <int FMT, bool L2, bool APPROX, int CTAS>
__global__ void __launch_bounds__(PAIR_THREADS, CTAS)
scan_finalize_kernel(const ScanFinalize p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SelectScratch sel;
    __shared__ __align__(16) uint64_t keys[SELECT_CAP];
    // (sorted results take the place of the selection's histogram and minima, which are done with by then: seven CTAs an SM)
    uint64_t* const best = reinterpret_cast<uint64_t*>(sel.hist);
    __shared__ uint32_t group_ids[APPROX ? FINAL_GROUPS : 1];
    __shared__ float part[PAIR_THREADS / 32];
    const PairScan& sc = p.scan;
    const uint64_t q = blockIdx.x;
    const uint32_t nprobe = sc.nprobe, dim = sc.s.dim;
    uint32_t* base_s = reinterpret_cast<uint32_t*>(smem);
    uint32_t* start_s = base_s + sc.nprobe;
    const bool plain = FMT == ROW_SQ8;
    float* qs = reinterpret_cast<float*>(smem + (2 * nprobe * sizeof(uint32_t) + 15) / 16 * 16);
    float* qc = qs + (plain ? (dim + 3) / 4 * 4 : 0u);     // SQ8: lower, then diff
    const uint32_t n = sc.t.rows[q];
    uint32_t* scores = reinterpret_cast<uint32_t*>(sc.t.scores + q * sc.t.stride);
    for (uint32_t i = threadIdx.x; i < nprobe; i += PAIR_THREADS) {
        const int32_t l = __ldg(sc.probes + q * nprobe + i);
        base_s[i] = __ldg(sc.t.base + q * nprobe + i);
        start_s[i] = l >= 0 && static_cast<uint32_t>(l) < sc.s.nlist ? __ldg(sc.s.list_off + l) : 0u;
    }
    if (plain) {
        const float* src = p.queries + q * dim;
        for (uint32_t d = threadIdx.x; d < dim; d += PAIR_THREADS) {
            qs[d] = __ldg(src + d);
            if (FMT == ROW_SQ8) {
                qc[d] = __ldg(p.lower + d);
                qc[dim + d] = __ldg(p.diff + d);
            }
        }
    }
    if (APPROX && FMT != ROW_SQ8) {
        stage_query<FMT>(sc, q, qc, PAIR_THREADS);
    }
    __syncthreads();
    const ScorePosition position{base_s, start_s, nprobe};
    auto exact = [&](uint32_t pos) -> float {
        const uint8_t* rec = sc.s.codes + static_cast<uint64_t>(pos) * sc.s.code_stride;
        if constexpr (FMT == ROW_SQ8) {
            return sq8_exact_distance(rec, dim, L2, qs, qc, qc + dim);
        } else {
            const float qn = FMT == ROW_RABITQ ? __ldg(sc.s.queries + q * (dim + 1) + dim) : 0.f;
            return record_exact_distance<FMT, L2>(rec, dim, sc.row_bytes, qc, qn);
        }
    };
    uint32_t found = 0, left = ORDERED_INF;   // left: no score that was not collected is below it
    bool selected = false;
    if (APPROX && sc.t.minima != nullptr) {
        // First the groups of 32 scores that can hold one of the kcand best: those whose smallest is not above the
        // kcand-th smallest minimum.  Then the scores of those groups alone.
        const uint32_t* minima = sc.t.minima + q * (sc.t.stride / 32);
        const uint32_t groups = n / 32;
        uint32_t upto;
        const uint32_t bound = block_bound<PAIR_THREADS>(load_source([&](uint32_t i) { return __ldg(minima + i); }), groups, p.kcand,
                                                         p.kcand + p.kcand / 8 + 8, sel, &upto);
        if (upto <= FINAL_GROUPS) {
            if (threadIdx.x == 0) {
                sel.count = 0;
            }
            __syncthreads();
            for (uint32_t i = threadIdx.x; i < groups; i += PAIR_THREADS) {
                if (__ldg(minima + i) <= bound) {
                    group_ids[atomicAdd(&sel.count, 1u)] = i;
                }
            }
            __syncthreads();
            const uint32_t m = sel.count;
            __syncthreads();
            const auto at = [&](uint32_t i) -> uint32_t { return group_ids[i >> 5] * 32 + (i & 31u); };
            const GroupPosition where{group_ids, position};
            found = block_select<PAIR_THREADS>(load_source([&](uint32_t i) { return ScoreSource<>::ordered(__ldg(scores + at(i))); }), where,
                                               m * 32, p.kcand, keys, sel, &left);
            // (the other groups' scores are above `bound`)
            left = groups > m ? min(left, bound) : left;
            selected = true;
        }
    }
    if (!selected) {
        found = block_select<PAIR_THREADS>(ScoreSource<>{scores}, position, n, p.kcand, keys, sel, &left);
    }
    if (p.rows_scanned != nullptr) {
        uint32_t rows = 0;
        for (uint32_t i = threadIdx.x; i < nprobe; i += PAIR_THREADS) {
            const int32_t l = __ldg(sc.probes + q * nprobe + i);
            rows += l >= 0 && static_cast<uint32_t>(l) < sc.s.nlist ? __ldg(sc.s.list_off + l + 1) - __ldg(sc.s.list_off + l) : 0u;
        }
        if (threadIdx.x == 0) {
            sel.total = 0;
        }
        __syncthreads();
        rows = __reduce_add_sync(0xffffffffu, rows);
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&sel.total, rows);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            p.rows_scanned[q] = sel.total;
        }
    }
    if (APPROX) {
        // Everything that was collected is re-scored, usually kcand rows and a third more: ordering them by score first, to drop
        // those, cost more than their distances.  (All of up to 256, and of rows that tie at the bound up to SELECT_CAP.  Cutting
        // those to kcand first: 1000 queries of 12,500 rows of 400 bits, one in fifty set, 38.4 ms for 38.1, since such a query
        // scores all its rows exactly below anyway; three hundred different rows of 96 bytes, 1.33 for 1.46.)
        const bool dropped = left < ORDERED_INF;   // (else every row with a score was collected)
        const float last = dropped ? ordered_to_float(left) : 0.f;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < found; i += PAIR_THREADS) {
            const uint32_t pos = static_cast<uint32_t>(keys[i]);
            keys[i] = make_key(exact(pos), pos);
        }
        block_sort_to<PAIR_THREADS>(keys, found, p.kscan, best);
        float margin, offset = 0.f;
        const float rows_max = __ldg(p.row_max);
        if constexpr (FMT == ROW_RABITQ) {
            const float qn = __ldg(sc.s.queries + q * (dim + 1) + dim);
            // the dropped parts of the int8 terms and the additions' rounding, through 2 |x| |q| / error
            const float ip = dim * (__ldg(sc.qscale + q) * (0.5f / 64516.0f) + 1.2e-7f);
            margin = 2.0f * qn * __ldg(p.row_max + 1) * ip + 1e-6f * (rows_max + qn) * (rows_max + qn);
        } else {
            float qq = 0.f, ss = 0.f;
            for (uint32_t d = threadIdx.x; d < dim; d += PAIR_THREADS) {
                const float v = FMT == ROW_SQ8 ? qs[d] : qc[d];
                qq = fmaf(v, v, qq);
                if (FMT == ROW_SQ8) {
                    const float span = fabsf(qc[d]) + fabsf(qc[dim + d]);
                    ss = fmaf(span, span, ss);
                }
            }
            qq = pair_block_sum(qq, part);
            const float qn = sqrtf(qq);
            const float kth = dropped && L2 ? ordered_to_float(static_cast<uint32_t>(best[p.kscan - 1] >> 32)) : 0.f;
            // Q, X and S are the norms of the query, of the longest row and of |lower| + |diff|, d the k-th distance.
            constexpr float EPS = 6.0e-8f;
            const float chain = EPS * static_cast<float>(dim + 16);   // rounding of a chain of dim products
            if constexpr (FMT == ROW_SQ8) {
                // The integer sums are exact, so what remains is what the terms leave out; the chains behind |x|^2 and the exact
                // distance (X^2 and d, or X Q); the query's constant, 256 partial sums; and the rounding of the dequantized
                // values and of the last few operations.  (One (dim + 16) 2^-23 of (Q + X + S)^2 for all of them was five
                // times as large: of 100 results among 390 rows a list, 960 dimensions, some queries of every batch were
                // never sure and scored all their rows, 5.9 ms instead of 0.3.)
                const float span = sqrtf(pair_block_sum(ss, part)), few = EPS * static_cast<float>(dim / PAIR_THREADS + 32);
                margin = 2.0f * dim * 128.0f * __ldg(sc.qscale + q) * (0.5f / 64516.0f);
                margin += L2 ? chain * (rows_max * rows_max + kth) + few * (qq + 2.0f * qn * span)
                             : chain * rows_max * qn + few * (1.0f + qn * span);
            } else {
                // The sums of the tensor cores (16 products and the running sum per step, cut one bit below fp32's last or
                // lower; fp32 rows: two steps into one accumulator, and three dropped products of 2^-18); the exact chain
                // (d, or X Q); the sums behind X^2 and Q^2, over 32 lanes or more.
                const float matrix = FMT == ROW_F32 ? 2.2f * chain + 3.0f / 262144.0f : 1.1f * chain;
                const float few = EPS * static_cast<float>(dim / 32 + 32), size = qn * rows_max;
                offset = L2 ? qq : 1.0f;
                margin = L2 ? chain * kth + 2.0f * matrix * size + few * (qq + rows_max * rows_max) : (chain + matrix) * size + 3e-7f;
            }
        }
        margin += 1e-30f;   // (products below the smallest normal number round absolutely)
        // A margin that is not finite: scores may have overflowed, and a row whose score is not a number is not among the
        // found although its distance may be small.
        const bool sure = margin < INFINITY &&
                          (!dropped || ordered_to_float(static_cast<uint32_t>(best[p.kscan - 1] >> 32)) < last + offset - margin);
        if (!sure && n > 0) {
            for (uint32_t i = threadIdx.x; i < n; i += PAIR_THREADS) {
                if (scores[i] != SCORE_FILTERED) {
                    scores[i] = __float_as_uint(exact(position(i)));
                }
            }
            __syncthreads();
            const volatile uint32_t* rescored = scores;
            found = block_select<PAIR_THREADS>(load_source([&](uint32_t i) { return ScoreSource<>::ordered(rescored[i]); }), position, n,
                                               p.kscan, keys, sel);
            block_sort_to<PAIR_THREADS>(keys, found, p.kscan, best);
        }
    } else {
        block_sort_to<PAIR_THREADS>(keys, found, p.kscan, best);
    }
    uint32_t have = min(found, p.kscan);
    if (p.rerank_ids != nullptr) {
        // the candidates of the rerank, by inner id; 0xFFFFFFFF = none
        for (uint32_t i = threadIdx.x; i < p.kscan; i += PAIR_THREADS) {
            p.rerank_ids[q * p.kscan + i] = i < have ? __ldg(p.pos_inner + static_cast<uint32_t>(best[i])) : 0xFFFFFFFFu;
        }
        return;
    }
    for (uint32_t i = threadIdx.x; i < p.k; i += PAIR_THREADS) {
        const bool there = i < have;
        const uint64_t key = there ? best[i] : KEY_INF;
        const uint32_t inner = there ? __ldg(p.pos_inner + static_cast<uint32_t>(key)) : 0u;
        p.ids[q * p.k + i] = there ? __ldg(p.labels + inner) : -1;
        p.dists[q * p.k + i] = there ? ordered_to_float(static_cast<uint32_t>(key >> 32)) : INFINITY;
    }
}

// FlattenReorder::Reorder (src/impl/reorder/flatten_reorder.cpp:76-118): the fp32 distance of every candidate, a warp
// per candidate (lanes stride the dimensions, partial sums meet in a tree), then the k best as results.  The bound is
// reading the candidates' rows from memory, so a query's candidates are spread over RERANK_PARTS CTAs with a whole
// row (1024 dimensions) requested at once per warp; the CTA that finishes a query last orders its distances.
constexpr uint32_t RERANK_PARTS = 4;

struct Rerank {
    const float* queries;
    const float* flat;         // [n x dim] rows by inner id
    uint32_t dim, ncand, k;
    const uint32_t* ids;       // [nq x ncand] inner ids, 0xFFFFFFFF = none
    uint64_t* keys;            // [nq x ncand]
    uint32_t* done;            // [nq] zero before and after
    const int64_t* labels;
    int64_t* out_ids;
    float* out_dists;
};

template <bool L2>
__global__ void __launch_bounds__(PAIR_THREADS)
rerank_rows_kernel(const Rerank p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ __align__(16) uint64_t keys[1024];
    __shared__ __align__(16) uint64_t best[1024];
    __shared__ uint32_t last;
    float* qs = reinterpret_cast<float*>(smem);
    const uint64_t q = blockIdx.x / RERANK_PARTS;
    const uint32_t part = blockIdx.x % RERANK_PARTS;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (uint32_t d = threadIdx.x; d < p.dim; d += PAIR_THREADS) {
        qs[d] = __ldg(p.queries + q * p.dim + d);
    }
    __syncthreads();
    for (uint32_t c = part * (PAIR_THREADS / 32) + warp; c < p.ncand; c += RERANK_PARTS * (PAIR_THREADS / 32)) {
        const uint32_t inner = __ldg(p.ids + q * p.ncand + c);
        uint64_t key = KEY_INF;
        if (inner != 0xFFFFFFFFu) {
            const float* x = p.flat + static_cast<uint64_t>(inner) * p.dim;
            float s = 0.f;
            for (uint32_t d0 = lane; d0 < p.dim; d0 += 1024) {
                float v[32];
#pragma unroll
                for (uint32_t u = 0; u < 32; ++u) {
                    v[u] = d0 + u * 32 < p.dim ? __ldg(x + d0 + u * 32) : 0.f;
                }
#pragma unroll
                for (uint32_t u = 0; u < 32; ++u) {
                    const uint32_t d = d0 + u * 32;
                    if (d < p.dim) {
                        if (L2) {
                            const float t = qs[d] - v[u];
                            s = fmaf(t, t, s);
                        } else {
                            s = fmaf(qs[d], v[u], s);
                        }
                    }
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                s += __shfl_xor_sync(0xffffffffu, s, o);
            }
            key = make_key(L2 ? s : 1.0f - s, inner);
        }
        if (lane == 0) {
            p.keys[q * p.ncand + c] = key;
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(p.done + q, 1u) == RERANK_PARTS - 1 ? 1u : 0u;
    }
    __syncthreads();
    if (last == 0) {
        return;
    }
    if (threadIdx.x == 0) {
        p.done[q] = 0;
    }
    __threadfence();
    __shared__ uint32_t have;
    if (threadIdx.x == 0) {
        have = 0;
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < p.ncand; i += PAIR_THREADS) {
        const uint64_t key = *reinterpret_cast<const volatile uint64_t*>(p.keys + q * p.ncand + i);
        if (key != KEY_INF) {
            keys[atomicAdd(&have, 1u)] = key;
        }
    }
    __syncthreads();
    const uint32_t n = have;
    block_sort_to<PAIR_THREADS>(keys, n, p.k, best);
    for (uint32_t i = threadIdx.x; i < p.k; i += PAIR_THREADS) {
        const bool there = i < n;
        p.out_ids[q * p.k + i] = there ? __ldg(p.labels + static_cast<uint32_t>(best[i])) : -1;
        p.out_dists[q * p.k + i] = there ? ordered_to_float(static_cast<uint32_t>(best[i] >> 32)) : INFINITY;
    }
}

}  // namespace vb200
