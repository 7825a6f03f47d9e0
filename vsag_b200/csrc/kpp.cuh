// k-means++ seeding as one persistent launch (KMeansCluster::select_initial_centroids_kmeans_plus_plus,
// src/impl/cluster/kmeans_cluster.cpp:383-435).
//
// The k rounds depend on one another, so a round's latency is what counts: as two launches per round it took 40 us
// for 64,000 x 96 rows (35 us of them waiting for rows that had to come from L2 again), 999 times.  Here every CTA
// keeps its share of the rows for all rounds -- in shared memory when they fit the chip together (about 29 MB), and of
// rows that have a thread each the first dimensions in registers, else streamed through it from L2 or memory.
//
// A round's two exchanges are words of 32 bits of data and the round's number, written and polled as they are: every
// CTA's partial sum, which every CTA reads, and the row that is picked, by the CTA that holds it.  (As two grid barriers, after
// which the sums, the pick and then its row were read, 7.05 us a round of 64,000 x 96 rows; 5.5 this way.)  The words of two
// rounds do not meet: a CTA writes its sum of round r + 2 when it has the row of round r + 1, to which every CTA's sum of that
// round belongs, written after it had read all sums of round r; there are two sets of them.  One warp of a CTA reads the sums: with
// a thread for each, 148 CTAs' polls of the same few lines held one another up.  So do the polls of four CTAs an SM, which the streamed form
// has, while some still wait for rows: there the sums are counted in, and one thread of a CTA polls the count and then the
// number of the row (a round of 285,015 x 145 rows: 48 us
// with grid barriers, 74 with polled sums, 42.6 this way).
#pragma once

#include "block_select.cuh"
#include "row_scan.cuh"

namespace vb200 {

// CTAs whose sums a lane of the first warp reads (streamed: a thread of the CTA); so the launch has 32 (RS_ROWS) times that many at most.
constexpr uint32_t KPP_RUN = 5;

// Counts this CTA's sum in and waits until all have been; false when they do not come.
__device__ __forceinline__ bool
kpp_count_in(unsigned long long* count, unsigned long long all, uint32_t limit) {
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(count) : "memory");
    for (uint32_t spin = 0; spin < limit; ++spin) {
        unsigned long long seen;
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(seen) : "l"(count) : "memory");
        if (seen >= all) {
            return true;
        }
    }
    return false;
}

__device__ __forceinline__ double
kpp_sum_of(const unsigned long long* at) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(at) : "memory");
    return v;
}

struct KppRounds {
    const float* x;
    uint64_t n;
    uint32_t dim, k;
    uint64_t per;                 // rows per CTA
    uint64_t first;               // the row picked in round 0
    const double* u;              // [k] the rounds' uniform draws (entry 0 unused)
    float* min_d;                 // [n] squared distance to the nearest centre (streamed form)
    unsigned long long* part;     // [2][grid][2] words of the partial sums (streamed: the sums, in [0]); zero before the launch
    unsigned long long* count;    // [1] sums counted in (streamed form); zero before the launch
    unsigned long long* row;      // [dim] words of the picked row (streamed: [0] its number); zero before the launch
    float* centroids;             // [k x dim]
    int64_t* picked;              // [k] or null
    uint32_t* state;              // [0] first round that found no row apart from the centres (0xFFFFFFFF: none)
    uint32_t* failed;             // set to 1 when a wait gave up
    uint32_t spin_limit;
};

__device__ __forceinline__ void
kpp_put(unsigned long long* at, uint32_t data, uint32_t round) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(at), "l"((static_cast<unsigned long long>(round) << 32) | data) : "memory");
}

// The word of this round; *ok = false when it does not come.
__device__ __forceinline__ uint32_t
kpp_get(const unsigned long long* at, uint32_t round, uint32_t limit, bool* ok) {
    for (uint32_t spin = 0; spin < limit; ++spin) {
        unsigned long long w;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(at) : "memory");
        if (static_cast<uint32_t>(w >> 32) == round) {
            return static_cast<uint32_t>(w);
        }
    }
    *ok = false;
    return 0;
}

// N partial sums of this round, two words each, zeros past the last of `left`.  All are asked for together: one after the other, each a trip to
// L2, five of them were 4 us of a round.
template <uint32_t N>
__device__ __forceinline__ bool
kpp_get_sums(const unsigned long long* at, uint32_t left, uint32_t round, uint32_t limit, double (&out)[N]) {
    for (uint32_t spin = 0; spin < limit; ++spin) {
        unsigned long long lo[N], hi[N];
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            lo[i] = hi[i] = static_cast<unsigned long long>(round) << 32;
            if (i < left) {
                asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(lo[i]), "=l"(hi[i]) : "l"(at + 2 * i) : "memory");
            }
        }
        bool all = true;
#pragma unroll
        for (uint32_t i = 0; i < N; ++i) {
            all = all && static_cast<uint32_t>(lo[i] >> 32) == round && static_cast<uint32_t>(hi[i] >> 32) == round;
            out[i] = __longlong_as_double(static_cast<long long>((hi[i] << 32) | (lo[i] & 0xFFFFFFFFull)));
        }
        if (all) {
            return true;
        }
    }
    return false;
}

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

// RESIDENT: rows in shared memory, [per][dim | 1] (an odd stride: a row per lane reads without conflicts).  REG > 0 (then
// per <= T): thread r holds the first REG dimensions of row r in registers, zeros past the last, so that a round reads the centre
// from shared memory and not the rows (433 rows of 96 dimensions are 1300 cycles of it).
// Dynamic shared memory: [RESIDENT: -, streamed: the stages] the centre (max(dim, REG) values, a multiple of 4), [RESIDENT] rows and
// their distances.
template <bool RESIDENT, int REG, int UNIT, int T>
__global__ void __launch_bounds__(T)
kpp_rounds_kernel(const KppRounds p) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ double scan[32];
    __shared__ double s_base, s_total, s_thr;
    __shared__ uint32_t s_owner;
    __shared__ unsigned long long s_row;
    const uint32_t dim = p.dim, stride = dim | 1u, qpad = max((dim + 3) / 4 * 4, static_cast<uint32_t>(REG)), grid = gridDim.x;
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
    // the first centre
    for (uint32_t d = threadIdx.x; d < qpad; d += T) {
        const float v = d < dim ? __ldg(p.x + p.first * dim + d) : 0.f;
        c[d] = v;
        if (d < dim && blockIdx.x == 0) {
            p.centroids[d] = v;
        }
    }
    if (threadIdx.x == 0 && blockIdx.x == 0 && p.picked != nullptr) {
        p.picked[0] = static_cast<int64_t>(p.first);
    }
    __syncthreads();
    float head[REG > 0 ? REG : 1];
    if (REG > 0) {
#pragma unroll
        for (uint32_t d = 0; d < REG; ++d) {
            head[d] = threadIdx.x < mine && d < dim ? rows[threadIdx.x * stride + d] : 0.f;
        }
    }
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr uint32_t RUN = KPP_RUN;
    bool ok = true;
    for (uint32_t round = 1; round < p.k; ++round) {
        // distances: difference, then one FMA per dimension in ascending order
        double acc = 0.0;
        if (REG > 0) {
            if (threadIdx.x < mine) {
                float s = 0.f;
#pragma unroll
                for (uint32_t d = 0; d < REG; d += 4) {
                    const float4 v = *reinterpret_cast<const float4*>(c + d);
                    float t = __fsub_rn(head[d], v.x);
                    s = fmaf(t, t, s);
                    t = __fsub_rn(head[d + 1], v.y);
                    s = fmaf(t, t, s);
                    t = __fsub_rn(head[d + 2], v.z);
                    s = fmaf(t, t, s);
                    t = __fsub_rn(head[d + 3], v.w);
                    s = fmaf(t, t, s);
                }
                const float* x = rows + threadIdx.x * stride;
#pragma unroll 8
                for (uint32_t d = REG; d < dim; ++d) {
                    const float t = __fsub_rn(x[d], c[d]);
                    s = fmaf(t, t, s);
                }
                const float m = s < md[threadIdx.x] ? s : md[threadIdx.x];
                md[threadIdx.x] = m;
                acc = static_cast<double>(m);
            }
        } else if (RESIDENT) {
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
        // the CTA's sum goes out first; its rows' running sums are formed while the other CTAs' sums come in
        {
            double v = acc;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                v += __shfl_xor_sync(0xffffffffu, v, o);
            }
            if (lane == 0) {
                scan[warp] = v;
            }
        }
        __syncthreads();
        unsigned long long* part = p.part + static_cast<size_t>(round & 1u) * grid * 2;
        if (!RESIDENT) {
            if (threadIdx.x == 0) {
                double v = 0.0;
                for (uint32_t w = 0; w < T / 32; ++w) {
                    v += scan[w];
                }
                asm volatile("st.relaxed.gpu.global.f64 [%0], %1;" ::"l"(part + blockIdx.x * 2), "d"(v) : "memory");
                ok = kpp_count_in(p.count, static_cast<unsigned long long>(round) * grid, p.spin_limit);
                s_owner = 0xFFFFFFFFu;
                s_row = ~0ull;
            }
            if (__syncthreads_or(ok ? 0 : 1) != 0) {
                break;
            }
            const uint32_t g0 = threadIdx.x * RUN;
            double in[RUN], local = 0.0;
#pragma unroll
            for (uint32_t i = 0; i < RUN; ++i) {
                in[i] = g0 + i < grid ? kpp_sum_of(part + (g0 + i) * 2) : 0.0;
            }
#pragma unroll
            for (uint32_t i = 0; i < RUN; ++i) {
                local += in[i];
            }
            const double upto = block_inclusive_sum_f64<T>(local, scan);
            if (threadIdx.x == T - 1) {
                s_total = upto;
                s_thr = upto * __ldg(p.u + round);
            }
            __syncthreads();
            // (every thread whose run ends at or past the threshold names the first CTA of its run that does; the least counts)
            uint32_t first = 0xFFFFFFFFu;
            double base = upto - local;
            if (upto >= s_thr && g0 < grid) {
#pragma unroll
                for (uint32_t i = 0; i < RUN; ++i) {
                    if (first == 0xFFFFFFFFu && g0 + i < grid) {
                        const double next = base + in[i];
                        if (next >= s_thr || i + 1 == RUN || g0 + i + 1 == grid) {
                            first = g0 + i;
                        } else {
                            base = next;
                        }
                    }
                }
                atomicMin(&s_owner, first);
            }
            __syncthreads();
            if (first != 0xFFFFFFFFu && first == s_owner) {
                s_base = base;
            }
        } else if (warp == 0) {
            double v = lane < T / 32 ? scan[lane] : 0.0;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                v += __shfl_xor_sync(0xffffffffu, v, o);
            }
            if (lane == 0) {
                const unsigned long long bits = static_cast<unsigned long long>(__double_as_longlong(v));
                kpp_put(part + blockIdx.x * 2, static_cast<uint32_t>(bits), round);
                kpp_put(part + blockIdx.x * 2 + 1, static_cast<uint32_t>(bits >> 32), round);
            }
            // the CTA in whose rows the running sum over all reaches the threshold, and the sum before it (the same in every CTA)
            const double u = __ldg(p.u + round);
            double in[RUN], local = 0.0;
            ok = kpp_get_sums<RUN>(part + lane * RUN * 2, lane * RUN < grid ? grid - lane * RUN : 0u, round, p.spin_limit, in);
#pragma unroll
            for (uint32_t i = 0; i < RUN; ++i) {
                local += in[i];
            }
            double upto = local;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double w = __shfl_up_sync(0xffffffffu, upto, o);
                if (lane >= static_cast<uint32_t>(o)) {
                    upto += w;
                }
            }
            const double total = __shfl_sync(0xffffffffu, upto, 31), thr = total * u;
            const uint32_t reached = __ballot_sync(0xffffffffu, upto >= thr && lane * RUN < grid);
            if (lane == 0) {
                s_total = total;
                s_thr = thr;
                s_owner = 0xFFFFFFFFu;
                s_row = ~0ull;
            }
            __syncwarp();
            if (reached != 0 && lane == static_cast<uint32_t>(__ffs(reached) - 1)) {
                double at = upto - local;
#pragma unroll
                for (uint32_t i = 0; i < RUN; ++i) {
                    const uint32_t g = lane * RUN + i;
                    if (s_owner == 0xFFFFFFFFu && g < grid) {
                        const double next = at + in[i];
                        if (next >= thr || i + 1 == RUN || g + 1 == grid) {
                            s_owner = g;
                            s_base = at;
                        }
                        at = next;
                    }
                }
            }
        }
        double sum = acc;   // (REG: a row per thread) the running sum of the CTA's rows
        if (REG > 0) {
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double w = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= static_cast<uint32_t>(o)) {
                    sum += w;
                }
            }
            double before = 0.0;
            for (uint32_t w = 0; w < warp; ++w) {
                before += scan[w];
            }
            sum += before;
        }
        if (__syncthreads_or(ok ? 0 : 1) != 0) {
            break;
        }
        if (!(s_total > 0.0)) {   // every row coincides with a chosen centre (the same in every CTA)
            if (blockIdx.x == 0 && threadIdx.x == 0) {
                p.state[0] = round;
            }
            return;
        }
        const double thr = s_thr;
        const bool holds = s_owner == blockIdx.x || (s_owner == 0xFFFFFFFFu && blockIdx.x == grid - 1);
        if (holds) {
            uint64_t pick = p.n - 1;   // the reference's default when the running sum never gets there (the last CTA holds it)
            if (s_owner == blockIdx.x) {
                // the first of this CTA's rows whose running sum reaches it; rounding may keep the sum just below: its last row
                double base = s_base;
                if (REG > 0) {
                    const uint32_t past = __ballot_sync(0xffffffffu, threadIdx.x < mine && base + sum >= thr);
                    if (past != 0 && lane == 0) {
                        atomicMin(&s_row, static_cast<unsigned long long>(row0 + warp * 32 + __ffs(past) - 1));
                    }
                    __syncthreads();
                } else {
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
                }
                pick = s_row != ~0ull ? s_row : row0 + mine - 1;
            }
            if (!RESIDENT && threadIdx.x == 0) {
                kpp_put(p.row, static_cast<uint32_t>(pick), round);
            }
            for (uint32_t d = threadIdx.x; d < dim; d += T) {
                const float v = RESIDENT ? rows[(pick - row0) * stride + d] : __ldg(p.x + pick * dim + d);
                if (RESIDENT) {
                    kpp_put(p.row + d, __float_as_uint(v), round);
                }
                c[d] = v;
                p.centroids[static_cast<uint64_t>(round) * dim + d] = v;
            }
            if (threadIdx.x == 0 && p.picked != nullptr) {
                p.picked[round] = static_cast<int64_t>(pick);
            }
        } else if (!RESIDENT) {
            if (threadIdx.x == 0) {
                s_row = kpp_get(p.row, round, p.spin_limit, &ok);
            }
            if (__syncthreads_or(ok ? 0 : 1) != 0) {
                break;
            }
            for (uint32_t d = threadIdx.x; d < dim; d += T) {
                c[d] = __ldg(p.x + s_row * dim + d);
            }
        } else {
            for (uint32_t d = threadIdx.x; d < dim; d += T) {
                c[d] = __uint_as_float(kpp_get(p.row + d, round, p.spin_limit, &ok));
            }
        }
        if (__syncthreads_or(ok ? 0 : 1) != 0) {
            break;
        }
    }
    if (!ok) {
        *p.failed = 1;
    }
}

}  // namespace vb200
