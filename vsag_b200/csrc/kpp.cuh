// k-means++ seeding as one persistent launch (KMeansCluster::select_initial_centroids_kmeans_plus_plus,
// src/impl/cluster/kmeans_cluster.cpp:383-435).
//
// The k rounds depend on one another, so a round's latency is what counts: as two launches per round it took 40 us
// for 64,000 x 96 rows (35 us of them waiting for rows that had to come from L2 again), 999 times.  Here every CTA
// keeps its share of the rows for all rounds -- in shared memory when they fit the chip together (about 29 MB), else
// streamed through it from L2 or memory -- and two grid barriers per round exchange the partial sums and the pick.
#pragma once

#include <cooperative_groups.h>

#include "block_select.cuh"
#include "row_scan.cuh"

namespace vb200 {

struct KppRounds {
    const float* x;
    uint64_t n;
    uint32_t dim, k;
    uint64_t per;                 // rows per CTA
    uint64_t first;               // the row picked in round 0
    const double* u;              // [k] the rounds' uniform draws (entry 0 unused)
    float* min_d;                 // [n] squared distance to the nearest centre (streamed form)
    double* part;                 // [grid]
    unsigned long long* pick;     // [1]
    float* centroids;             // [k x dim]
    int64_t* picked;              // [k] or null
    uint32_t* state;              // [0] first round that found no row apart from the centres (0xFFFFFFFF: none)
};

// Inclusive prefix sum of a double per thread; `part` is a scratch of 32 doubles.
template <int T>
__device__ __forceinline__ double
block_inclusive_sum_f64(double v, double* part) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= static_cast<uint32_t>(o)) {
            v += u;
        }
    }
    __syncthreads();
    if (lane == 31) {
        part[warp] = v;
    }
    __syncthreads();
    for (uint32_t w = 0; w < warp; ++w) {
        v += part[w];
    }
    return v;
}

// RESIDENT: rows in shared memory, [per][dim | 1] (an odd stride: a row per lane reads without conflicts).
template <bool RESIDENT, int UNIT, int T>
__global__ void __launch_bounds__(T)
kpp_rounds_kernel(const KppRounds p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double scan[32];
    __shared__ double s_base;
    __shared__ uint32_t s_owner;
    __shared__ unsigned long long s_row;
    namespace cg = cooperative_groups;
    cg::grid_group grid = cg::this_grid();
    const uint32_t dim = p.dim, stride = dim | 1u, qpad = (dim + 3) / 4 * 4;
    float* c = RESIDENT ? reinterpret_cast<float*>(smem) : reinterpret_cast<float*>(smem + RS_STAGES * RS_STAGE);
    float* rows = c + qpad;
    const uint64_t row0 = blockIdx.x * p.per;
    const uint64_t mine = row0 < p.n ? (p.n - row0 < p.per ? p.n - row0 : p.per) : 0;
    float* md = RESIDENT ? rows + p.per * stride : p.min_d + row0;
    if (RESIDENT) {
        for (uint64_t e = threadIdx.x; e < mine * dim; e += T) {
            rows[e / dim * stride + e % dim] = __ldg(p.x + row0 * dim + e);
        }
    }
    for (uint64_t r = threadIdx.x; r < mine; r += T) {
        md[r] = 3.402823466e+38f;
    }
    __syncthreads();
    uint64_t last = p.first;
    for (uint32_t round = 1; round <= p.k; ++round) {
        // the centre picked last, into shared memory and -- by one CTA -- to the result
        for (uint32_t d = threadIdx.x; d < qpad; d += T) {
            const float v = d < dim ? __ldg(p.x + last * dim + d) : 0.f;
            c[d] = v;
            if (d < dim && blockIdx.x == round % gridDim.x) {
                p.centroids[static_cast<uint64_t>(round - 1) * dim + d] = v;
            }
        }
        if (threadIdx.x == 0 && p.picked != nullptr && blockIdx.x == round % gridDim.x) {
            p.picked[round - 1] = static_cast<int64_t>(last);
        }
        if (round == p.k) {
            return;
        }
        __syncthreads();
        // distances: difference, then one FMA per dimension in ascending order
        double acc = 0.0;
        if (RESIDENT) {
            for (uint32_t r = threadIdx.x; r < mine; r += T) {
                const float* x = rows + r * stride;
                float s = 0.f;
#pragma unroll 8
                for (uint32_t d = 0; d < dim; ++d) {
                    const float t = __fsub_rn(x[d], c[d]);
                    s = fmaf(t, t, s);
                }
                const float m = s < md[r] ? s : md[r];
                md[r] = m;
                acc += static_cast<double>(m);
            }
        } else if (mine > 0) {
            RowAcc<ROW_F32, true, 1> dist;
            row_stream<UNIT>(reinterpret_cast<const unsigned char*>(p.x + row0 * dim), static_cast<uint64_t>(dim) * 4, dim * 4, dim, mine, 0,
                             1, smem, c, qpad, dist, [&](uint64_t r, bool valid) {
                                 if (valid) {
                                     const float s = dist.acc[0], old = md[r];
                                     const float m = s < old ? s : old;
                                     md[r] = m;
                                     acc += static_cast<double>(m);
                                 }
                             });
        }
        const double sum = block_inclusive_sum_f64<T>(acc, scan);
        if (threadIdx.x == T - 1) {
            p.part[blockIdx.x] = sum;
        }
        grid.sync();
        // every CTA finds the CTA in whose rows the running sum reaches the threshold
        const uint32_t run = (gridDim.x + T - 1) / T, g0 = threadIdx.x * run;
        double local = 0.0;
        for (uint32_t g = g0; g < g0 + run && g < gridDim.x; ++g) {
            local += *reinterpret_cast<const volatile double*>(p.part + g);
        }
        const double upto = block_inclusive_sum_f64<T>(local, scan);
        if (threadIdx.x == T - 1) {
            s_base = upto;
            s_owner = 0xFFFFFFFFu;
            s_row = ~0ull;
        }
        __syncthreads();
        const double total = s_base;
        if (!(total > 0.0)) {   // every row coincides with a chosen centre (the same in every CTA)
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                p.state[0] = round;
            }
            return;
        }
        const double thr = total * __ldg(p.u + round);
        __syncthreads();
        // (every thread whose run ends at or past the threshold names the first CTA of its run that does; the least counts)
        if (upto >= thr && g0 < gridDim.x) {
            double at = upto - local;
            for (uint32_t g = g0; g < g0 + run && g < gridDim.x; ++g) {
                const double next = at + *reinterpret_cast<const volatile double*>(p.part + g);
                if (next >= thr || g + 1 == g0 + run || g + 1 == gridDim.x) {
                    atomicMin(&s_owner, g);
                    if (g == blockIdx.x) {
                        s_base = at;
                    }
                    break;
                }
                at = next;
            }
        }
        __syncthreads();
        if (s_owner == blockIdx.x) {
            // the first of this CTA's rows whose running sum reaches it; rounding may keep the sum just below: its last row
            double base = s_base;
            for (uint64_t r0 = 0; r0 < mine; r0 += T) {
                const uint64_t r = r0 + threadIdx.x;
                const double at = base + block_inclusive_sum_f64<T>(r < mine ? static_cast<double>(md[r]) : 0.0, scan);
                if (r < mine && at >= thr) {
                    atomicMin(&s_row, static_cast<unsigned long long>(row0 + r));
                }
                __syncthreads();
                if (s_row != ~0ull) {
                    break;
                }
                if (threadIdx.x == T - 1) {
                    s_base = at;
                }
                __syncthreads();
                base = s_base;
                __syncthreads();
            }
            if (threadIdx.x == 0) {
                *p.pick = s_row != ~0ull ? s_row : static_cast<unsigned long long>(row0 + mine - 1);
            }
        } else if (s_owner == 0xFFFFFFFFu && blockIdx.x == 0 && threadIdx.x == 0) {
            *p.pick = p.n - 1;   // the reference's default when the running sum never gets there
        }
        grid.sync();
        last = *reinterpret_cast<const volatile unsigned long long*>(p.pick);
    }
}

}  // namespace vb200
