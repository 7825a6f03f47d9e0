// Exact selection of the k smallest of n values by one CTA, without sorting the n values.
//
// What bounds it is the passes over the values, so it makes two: the first keeps one minimum per group of a
// few values (groups interleave, so that neighbouring values land in different groups), and the k-th smallest
// of those minima is an upper bound of the k-th smallest value, because the minima are k distinct values.  With
// two or more groups per wanted value the bound lets through about 1.3 k values; the second pass collects
// those, and only they are sorted.  Values that tie or crowd in such a way that the collection does not fit are
// narrowed down by histograms over the ordered bit patterns until it does.
#pragma once

#include "common.cuh"

namespace vb200 {

constexpr uint32_t ORDERED_INF = 0xFF800000u;     // float_to_ordered(+inf): larger patterns are NaNs, never selected
constexpr uint32_t SELECT_BINS = 1024;
constexpr uint32_t SELECT_GROUPS = 1024;          // group minima kept at most
constexpr uint32_t SELECT_CAP = 2048;             // values collected at most
constexpr uint32_t SELECT_RANKED = 256;           // keys sorted by counting, at most

struct alignas(16) SelectScratch {
    uint32_t hist[SELECT_BINS];
    uint32_t minima[SELECT_GROUPS];   // per group; the second pass reads them again
    uint32_t warp_part[32];
    uint32_t lo, hi, total, pick, upto, before, count;
};

// Inclusive prefix sum over the T threads of the CTA; every thread calls it, `part` is a scratch of 32 words.
template <int T>
__device__ __forceinline__ uint32_t
block_inclusive_sum(uint32_t v, uint32_t* part) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= static_cast<uint32_t>(o)) {
            v += u;
        }
    }
    __syncthreads();
    if (lane == 31) {
        part[warp] = v;
    }
    __syncthreads();
    uint32_t add = 0;
#pragma unroll
    for (int w = 0; w < T / 32; ++w) {
        add += static_cast<uint32_t>(w) < warp ? part[w] : 0u;
    }
    return v + add;
}

// A source hands out n ordered values: at(i) is value number i; walk calls visit(i, value) for a share of the
// numbers, thread `first` of `step`, such that the shares of first = 0 .. step-1 cover every number once.  The
// loads of several values are issued together: a thread waits for memory once per batch.
template <typename Load>
struct LoadSource {   // any load(i)
    Load load;
    __device__ __forceinline__ uint32_t
    at(uint32_t i) const {
        return load(i);
    }
    template <typename Visit>
    __device__ __forceinline__ void
    walk(uint32_t first, uint32_t step, uint32_t n, Visit visit) const {
        uint32_t i = first;
        for (; i < n && n - i > 7 * step; i += 8 * step) {
            uint32_t u[8];
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                u[j] = load(i + j * step);
            }
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                visit(i + j * step, u[j]);
            }
        }
        for (; i < n; i += step) {
            visit(i, load(i));
        }
    }
};

template <typename Load>
__device__ __forceinline__ LoadSource<Load>
load_source(Load load) {
    return LoadSource<Load>{load};
}

// Scores in memory, 16-byte aligned and readable up to a multiple of four.
template <bool SKIP_INF = false>
struct ScoreSource {
    const uint32_t* scores;   // fp32 bit patterns
    __device__ __forceinline__ static uint32_t
    ordered(uint32_t b) {
        const uint32_t u = (b & 0x80000000u) ? ~b : (b | 0x80000000u);   // float_to_ordered
        return SKIP_INF && u == ORDERED_INF ? 0xFFFFFFFFu : u;
    }
    __device__ __forceinline__ uint32_t
    at(uint32_t i) const {
        return ordered(__ldg(scores + i));
    }
    template <typename Visit>
    __device__ __forceinline__ void
    walk(uint32_t first, uint32_t step, uint32_t n, Visit visit) const {
        const uint32_t n4 = (n + 3) / 4;
        const uint4* v = reinterpret_cast<const uint4*>(scores);
        for (uint32_t i = first; i < n4; i += 4 * step) {
            uint4 u[4];
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                u[j] = i + j * step < n4 ? __ldg(v + i + j * step) : make_uint4(0x7FFFFFFFu, 0x7FFFFFFFu, 0x7FFFFFFFu, 0x7FFFFFFFu);
            }
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                const uint32_t at4 = 4 * (i + j * step);
                const uint32_t w[4] = {u[j].x, u[j].y, u[j].z, u[j].w};
#pragma unroll
                for (uint32_t c = 0; c < 4; ++c) {
                    if (at4 + c < n) {
                        visit(at4 + c, ordered(w[c]));
                    }
                }
            }
        }
    }
};

// An ordered value t such that at least k of the n values are <= t, and at most `cap` unless more than that
// tie at t exactly.  *upto = how many are <= t.  Values above ORDERED_INF do not take part; with fewer than k
// taking part, t = ORDERED_INF.
template <int T, typename Source>
__device__ uint32_t
block_bound(const Source& src, uint32_t n, uint32_t k, uint32_t cap, SelectScratch& s, uint32_t* upto) {
    uint32_t mn = 0xFFFFFFFFu, mx = 0, have = 0;
    src.walk(threadIdx.x, T, n, [&](uint32_t, uint32_t u) {
        if (u <= ORDERED_INF) {
            mn = min(mn, u);
            mx = max(mx, u);
            ++have;
        }
    });
    __syncthreads();
    if (threadIdx.x == 0) {
        s.lo = 0xFFFFFFFFu;
        s.hi = 0;
        s.total = 0;
    }
    __syncthreads();
    mn = __reduce_min_sync(0xffffffffu, mn);
    mx = __reduce_max_sync(0xffffffffu, mx);
    have = __reduce_add_sync(0xffffffffu, have);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&s.lo, mn);
        atomicMax(&s.hi, mx);
        atomicAdd(&s.total, have);
    }
    __syncthreads();
    uint32_t lo = s.lo, hi = s.hi, below = 0;
    if (s.total <= k) {
        *upto = s.total;
        return ORDERED_INF;
    }
    for (;;) {
        const uint32_t range = hi - lo;
        const uint32_t shift = range < SELECT_BINS ? 0u : static_cast<uint32_t>(22 - __clz(range));   // range >> shift < 1024
        for (uint32_t b = threadIdx.x; b < SELECT_BINS; b += T) {
            s.hist[b] = 0;
        }
        __syncthreads();
        src.walk(threadIdx.x, T, n, [&](uint32_t, uint32_t u) {
            if (u >= lo && u <= hi) {
                atomicAdd(&s.hist[(u - lo) >> shift], 1u);
            }
        });
        __syncthreads();
        constexpr int PER = SELECT_BINS / T;
        uint32_t c[PER], sum = 0;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            c[j] = s.hist[threadIdx.x * PER + j];
            sum += c[j];
        }
        const uint32_t incl = block_inclusive_sum<T>(sum, s.warp_part);
        uint32_t run = below + incl - sum;
        if (run < k && run + sum >= k) {
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                if (run < k && run + c[j] >= k) {
                    s.pick = threadIdx.x * PER + j;
                    s.upto = run + c[j];
                    s.before = run;
                }
                run += c[j];
            }
        }
        __syncthreads();
        const uint32_t bin = s.pick, reached = s.upto, before = s.before;
        __syncthreads();
        const uint32_t bin_lo = lo + (bin << shift);
        const uint32_t last = bin_lo + ((1u << shift) - 1u);
        if (reached <= cap || shift == 0) {
            *upto = reached;
            return min(last, hi);
        }
        below = before;
        hi = min(last, hi);
        lo = bin_lo;
    }
}

// The k smallest of the n values (ties: smallest payload first) among a few more, unsorted, as
// (value << 32 | payload(i)) in keys[SELECT_CAP]; returns how many were collected (>= k when that many take
// part, <= SELECT_CAP).  k <= 1024.  Every value is read once, and
// the groups of the smallest ones again.  *least_left (optional): no value that was not collected is below it; ORDERED_INF: every
// value that takes part was collected.
template <int T, typename Source, typename Payload>
__device__ uint32_t
block_select(const Source& src, const Payload& payload, uint32_t n, uint32_t k, uint64_t* keys, SelectScratch& s,
             uint32_t* least_left = nullptr) {
    uint32_t bound = ORDERED_INF;
    bool counted = false;
    uint32_t grouped = 0;   // how many groups have their minimum in s.minima
    if (n > 256 && n > k) {
        // groups: T threads times a power of two, two or more per wanted value as far as they go
        uint32_t per = 1;
        while (per * T < 2 * k && per * 2 * T <= SELECT_GROUPS) {
            per <<= 1;
        }
        const uint32_t groups = per * T;
        if (4 * k <= 3 * groups) {
            for (uint32_t g = 0; g < per; ++g) {
                uint32_t mn = 0xFFFFFFFFu;
                src.walk(g * T + threadIdx.x, groups, n, [&](uint32_t, uint32_t u) { mn = min(mn, u); });
                s.minima[g * T + threadIdx.x] = mn;
            }
            grouped = groups;
            __syncthreads();
            uint32_t upto;
            bound = block_bound<T>(load_source([&](uint32_t i) { return s.minima[i]; }), groups, k, k + k / 8 + 8, s, &upto);
        } else {
            uint32_t upto;
            bound = block_bound<T>(src, n, k, SELECT_CAP, s, &upto);
            counted = upto <= SELECT_CAP;
        }
    }
    auto collect = [&](uint32_t t, bool strict) -> uint32_t {
        __syncthreads();
        if (threadIdx.x == 0) {
            s.count = 0;
        }
        __syncthreads();
        auto take = [&](uint32_t i, uint32_t u) {
            if (u <= ORDERED_INF && (strict ? u < t : u <= t)) {
                const uint32_t slot = atomicAdd(&s.count, 1u);
                if (slot < SELECT_CAP) {
                    keys[slot] = (static_cast<uint64_t>(u) << 32) | payload(i);
                }
            }
        };
        // A thread reads its groups again only if their minimum passes: a few more than k of them do.  Worth it while those
        // are a third at most, and a group is sixteen values or more (1000 x 100k scores, k 26: 184 -> 174 us; 72 of 4096
        // scores: 120 -> 111 us with what follows; 416 of 1024 groups: 251 -> 270 us, so not there).
        if (3 * k <= grouped && n >= 16 * grouped) {
            for (uint32_t g = threadIdx.x; g < grouped; g += T) {
                if (s.minima[g] <= t) {
                    src.walk(g, grouped, n, take);
                }
            }
        } else {
            src.walk(threadIdx.x, T, n, take);
        }
        __syncthreads();
        return s.count;
    };
    uint32_t count = collect(bound, false);
    if (least_left != nullptr) {
        *least_left = bound;
    }
    if (count <= SELECT_CAP || counted) {
        return count;
    }
    uint32_t upto;
    bound = block_bound<T>(src, n, k, SELECT_CAP, s, &upto);
    if (least_left != nullptr) {
        *least_left = bound;
    }
    if (upto <= SELECT_CAP) {
        return collect(bound, false);
    }
    // more values tie at the k-th than fit: everything below it, then the ties with the smallest payloads
    const uint32_t below = collect(bound, true);
    uint32_t ties;
    const uint32_t last = block_bound<T>(
        load_source([&](uint32_t i) { return src.at(i) == bound ? min(payload(i), ORDERED_INF) : 0xFFFFFFFFu; }), n, k - below, k - below, s, &ties);
    for (uint32_t i = threadIdx.x; i < n; i += T) {
        if (src.at(i) == bound) {
            const uint32_t p = payload(i);
            if (p <= last) {
                const uint32_t slot = atomicAdd(&s.count, 1u);
                if (slot < SELECT_CAP) {
                    keys[slot] = (static_cast<uint64_t>(bound) << 32) | p;
                }
            }
        }
    }
    __syncthreads();
    return min(s.count, SELECT_CAP);
}

// Sorts `count` distinct keys and leaves the `keep` smallest, ascending, in out (a different buffer).  Up to 256
// keys every thread counts how many are smaller than its own, one pass and one barrier instead of a sorting
// network's many; more go through the network, whose instructions grow more slowly (464 keys: 27,000 a warp's share against
// 4,300; keys must then have room for the next power of two).
template <int T>
__device__ __forceinline__ void
block_sort_to(uint64_t* keys, uint32_t count, uint32_t keep, uint64_t* out) {
    __syncthreads();
    if (count <= SELECT_RANKED) {
        for (uint32_t i = threadIdx.x; i < count; i += T) {
            const uint64_t mine = keys[i];
            uint32_t rank = 0;
#pragma unroll 8
            for (uint32_t j = 0; j < count; ++j) {
                rank += keys[j] < mine ? 1u : 0u;
            }
            if (rank < keep) {
                out[rank] = mine;
            }
        }
        __syncthreads();
        return;
    }
    const uint32_t n2 = next_pow2(count);
    for (uint32_t i = count + threadIdx.x; i < n2; i += T) {
        keys[i] = KEY_INF;
    }
    block_bitonic_sort(keys, n2);
    for (uint32_t i = threadIdx.x; i < keep && i < count; i += T) {
        out[i] = keys[i];
    }
    __syncthreads();
}

// ---- the same by one warp -----------------------------------------------------------------------------------
// For a few dozen values out of some thousands a CTA spends most of its time in its forty barriers; a warp has none, keeps the
// group minima in registers and finds the bound by halving the range of values in question (a count over the registers and one
// reduction per step).
constexpr uint32_t WARP_SELECT_MAX = 128;    // wanted at most
constexpr uint32_t WARP_SELECT_CAP = 256;    // collected at most

// Bitonic sort of 32 * R keys held R per lane (element e = 32 * r + lane lives in key[r] of lane e % 32):
// compare-exchanges inside a lane when the partner is 32 or more elements away, shuffles otherwise; ascending.
template <int R>
__device__ __forceinline__ void
warp_sort_registers(uint64_t (&key)[R], uint32_t lane) {
#pragma unroll
    for (uint32_t size = 2; size <= 32u * R; size <<= 1) {
#pragma unroll
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= 32) {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int pr = r ^ static_cast<int>(stride >> 5);
                    if (pr > r) {
                        const bool up = (((static_cast<uint32_t>(r) << 5) | lane) & size) == 0;
                        const uint64_t a = key[r], b = key[pr];
                        if ((a > b) == up) {
                            key[r] = b;
                            key[pr] = a;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const uint32_t e = (static_cast<uint32_t>(r) << 5) | lane;
                    const uint64_t mine = key[r];
                    const uint64_t other = __shfl_xor_sync(0xffffffffu, mine, stride);
                    const bool up = (e & size) == 0;
                    const bool lower = (lane & stride) == 0;
                    const bool take_min = lower == up;
                    key[r] = take_min ? (mine < other ? mine : other) : (mine > other ? mine : other);
                }
            }
        }
    }
}

// buf[0 .. 32 R) sorted ascending through registers (one warp).
template <int R>
__device__ __noinline__ void
warp_sort_buffer(uint64_t* buf, uint32_t lane) {
    uint64_t key[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        key[r] = buf[r * 32 + lane];
    }
    warp_sort_registers<R>(key, lane);
#pragma unroll
    for (int r = 0; r < R; ++r) {
        buf[r * 32 + lane] = key[r];
    }
    __syncwarp();
}

// Visits the n values of load(i) in order, 32 at a time with eight loads of a lane together: visit(i, value), value 0xFFFFFFFF for i >= n.
template <typename Load, typename Visit>
__device__ __forceinline__ void
warp_walk(const Load& load, uint32_t n, uint32_t lane, Visit visit) {
    for (uint32_t i0 = 0; i0 < n; i0 += 256) {
        uint32_t u[8];
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            const uint32_t i = i0 + j * 32 + lane;
            u[j] = i < n ? load(i) : 0xFFFFFFFFu;
        }
#pragma unroll
        for (uint32_t j = 0; j < 8; ++j) {
            if (i0 + j * 32 < n) {
                visit(i0 + j * 32 + lane, u[j], j);
            }
        }
    }
}

// The smallest value in m[] of all lanes that `k` of them are at or below, or one a few ranks above it; ORDERED_INF when no more than k
// are numbers.
template <int PER>
__device__ __forceinline__ uint32_t
warp_bound(const uint32_t (&m)[PER], uint32_t k) {
    uint32_t low = 0xFFFFFFFFu, high = 0, have = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
        if (m[j] <= ORDERED_INF) {
            low = min(low, m[j]);
            high = max(high, m[j]);
            ++have;
        }
    }
    low = __reduce_min_sync(0xffffffffu, low);
    high = __reduce_max_sync(0xffffffffu, high);
    have = __reduce_add_sync(0xffffffffu, have);
    if (have <= k) {
        return ORDERED_INF;
    }
    while (low < high) {   // `k` values are at or below `high`, fewer are below `low`
        const uint32_t mid = low + (high - low) / 2;
        uint32_t count = 0;
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            count += m[j] <= mid ? 1u : 0u;
        }
        count = __reduce_add_sync(0xffffffffu, count);
        if (count < k) {
            low = mid + 1;
        } else {
            high = mid;
            if (count <= k + k / 16) {
                break;
            }
        }
    }
    return high;
}

// Values of load(0 .. n) at or below t, as (value << 32 | payload(i)) in keys[WARP_SELECT_CAP]; how many there are (more than fit: the
// first ones are there).
template <typename Load, typename Payload>
__device__ __forceinline__ uint32_t
warp_collect(const Load& load, const Payload& payload, uint32_t n, uint32_t t, uint64_t* keys, uint32_t lane) {
    uint32_t count = 0;
    warp_walk(load, n, lane, [&](uint32_t i, uint32_t u, uint32_t) {
        const bool take = u <= t && u <= ORDERED_INF;
        const uint32_t mask = __ballot_sync(0xffffffffu, take);
        if (mask != 0) {
            const uint32_t at = count + __popc(mask & ((1u << lane) - 1u));
            if (take && at < WARP_SELECT_CAP) {
                keys[at] = (static_cast<uint64_t>(u) << 32) | payload(i);
            }
            count += __popc(mask);
        }
    });
    __syncwarp();
    return count;
}

// A few more than the k smallest of the n values, unsorted in keys[WARP_SELECT_CAP]; how many, or more than WARP_SELECT_CAP when too many
// crowd at the k-th.  No value that was not collected is below *left (ORDERED_INF: all were collected).  k <= WARP_SELECT_MAX.
template <typename Load, typename Payload>
__device__ __forceinline__ uint32_t
warp_select(const Load& load, const Payload& payload, uint32_t n, uint32_t k, uint64_t* keys, uint32_t lane, uint32_t* left) {
    uint32_t t;
    if (k <= 40) {   // 128 groups: three or more per wanted value
        uint32_t m[4] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu};
        warp_walk(load, n, lane, [&](uint32_t, uint32_t u, uint32_t j) { m[j & 3u] = min(m[j & 3u], u); });
        t = n <= k ? ORDERED_INF : warp_bound(m, k);
    } else {         // 256, two or more
        uint32_t m[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            m[j] = 0xFFFFFFFFu;
        }
        warp_walk(load, n, lane, [&](uint32_t, uint32_t u, uint32_t j) { m[j & 7u] = min(m[j & 7u], u); });
        t = n <= k ? ORDERED_INF : warp_bound(m, k);
    }
    *left = t;
    return warp_collect(load, payload, n, t, keys, lane);
}

// keys[0 .. count) ascending, count <= WARP_SELECT_CAP (one warp).
__device__ __forceinline__ void
warp_sort(uint64_t* keys, uint32_t count, uint32_t lane) {
    const uint32_t padded = count <= 32 ? 32u : (count <= 64 ? 64u : (count <= 128 ? 128u : 256u));
    for (uint32_t i = count + lane; i < padded; i += 32) {
        keys[i] = KEY_INF;
    }
    __syncwarp();
    if (padded == 32) {
        warp_sort_buffer<1>(keys, lane);
    } else if (padded == 64) {
        warp_sort_buffer<2>(keys, lane);
    } else if (padded == 128) {
        warp_sort_buffer<4>(keys, lane);
    } else {
        warp_sort_buffer<8>(keys, lane);
    }
}

}  // namespace vb200
