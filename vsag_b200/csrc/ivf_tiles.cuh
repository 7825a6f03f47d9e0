// List scan of a batch as tensor-core tiles that write scores.
//
// A work item is one inverted list against up to 64 (32, 16) of the queries that probe it: the rows are read once
// for all of them, 128 at a time, and a tile [128 rows x queries] of inner products comes out of tcgen05.mma.  The
// epilogue turns each into a ranking score and stores it where the query's scores go (ivf_pairs.cuh); a CTA per
// query then selects, re-scores its candidates in the reference's operation order and checks that the margin
// between what it kept and what it dropped covers the tile arithmetic's error (otherwise it scores all its rows
// exactly).  Nothing is selected here, so no bounds, no buffers and no second phase are needed, and the kernel's
// time is that of reading the lists once (a few percent of them are probed by more queries than one item holds).
//
// Every role of the CTA runs on warps of its own and is a few steps ahead of the one it feeds: one takes items from
// the queue and copies rows, four gather the next item's queries, eight convert where the codec needs it, one thread
// issues the MMAs, eight warps drain them.  (With the loads, the conversions and the gathering of an item on the same
// warps, and the item's constants read by the epilogue, the kernel waited for one latency after another: 390 to
// 560 us instead of 279 for 1000 queries against 32 lists each of 500k x 128 fp32.)  How rows become operands:
//   fp32        two bf16 terms x = hi + lo, made in place in shared memory, which a tile waits for, or from the second batch after
//               the rows changed on read from a copy that holds them, where there is memory for one (280 us of the case
//               above, 173 from the copy, which takes 100 to make and as much memory as the rows); hi*hi + lo*hi and hi*lo are accumulated (the dropped terms are below 2^-16 |x||q|)
//   bf16, fp16  the codes as they are (TMA with the 128-byte swizzle); every product is exact in fp32
//   sq8         the tiled copy of the codes as signed bytes code - 128, against three int8 terms of the query's
//               weights: exact int32 sums
//   rabitq      the sign bits as bytes 0 / 1, spread in shared memory, against three int8 terms of the query; sum over
//               set bits = (sum of all terms + signed sum) / 2
#pragma once

#include <cuda.h>   // CUtensorMap

#include "ivf_pairs.cuh"
#include "ivf_scan_tc.cuh"

namespace vb200 {

constexpr int TILE_QUERY_WARPS = 4;
constexpr int TILE_CONV_WARPS = 8;
constexpr uint32_t TILE_PIECE = 128;                        // operand bytes per row and piece
constexpr uint32_t TILE_A_TERM = 128 * TILE_PIECE;          // 16 KiB
constexpr uint32_t TILE_MAX_STAGES = 8;
constexpr uint32_t TILE_DESCS = 4;                          // items described ahead
constexpr uint32_t TILE_ACC_COLS = 256;                     // tensor-memory columns per accumulator, two of them

// How a codec becomes MMA operands.
template <int FMT>
struct TileFmt {
    static constexpr bool INT8 = FMT == ROW_SQ8 || FMT == ROW_RABITQ;
    static constexpr bool SPLIT = FMT == ROW_F32 || FMT == ROW_F32_SPLIT;
    static constexpr bool CONVERT = FMT == ROW_F32 || FMT == ROW_RABITQ;
    static constexpr uint32_t A_TERMS = SPLIT ? 2 : 1;
    static constexpr uint32_t B_TERMS = INT8 ? 3 : (SPLIT ? 2 : 1);
    static constexpr uint32_t PIECE_DIMS = INT8 ? 128 : 64;
    static constexpr uint32_t STAGE = A_TERMS * TILE_A_TERM;
    // Warps by role: the first EPI drain accumulators, then one issues the MMAs, one copies rows, TILE_QUERY_WARPS gather queries,
    // TILE_CONV_WARPS convert.  Of sixteen draining warps four share the columns of 32 rows: 173 us for the split fp32 rows of the
    // case above; integer sums take more instructions a column and are no faster for it (109 against 123 us).
    static constexpr int EPI = CONVERT || INT8 ? 8 : 16;
    static constexpr int THREADS = 32 * (EPI + 2 + TILE_QUERY_WARPS + (CONVERT ? TILE_CONV_WARPS : 0));
};

// Lists of very different lengths are the rule (a list that many queries probe is often a long one): an item is at
// most TILE_SEGMENT rows of a list, so that no CTA is left with one long list at the end.
constexpr uint32_t TILE_SEGMENT = 1024;

struct alignas(16) TileItem {
    uint32_t lbeg, len, pair0, nqt;   // rows lbeg .. lbeg + len against pairs pair0 .. pair0 + nqt
    uint32_t row0, goff, pad0, pad1;  // their number within the list, and their first 8-row group (SQ8)
};

struct alignas(16) TilePair {
    uint32_t q, pad;
    uint64_t out;                     // where the scores of the (query, list) pair begin
};

struct TileScan {
    CUtensorMap map;            // the stored rows, or their bf16 terms (not SQ8)
    ScanParams s;               // constants; queries (RaBitQ: processed)
    PairTable t;
    const TileItem* items;
    uint32_t* queue;            // [0] number of items, [1] the next one to take
    const TilePair* pairs;      // grouped by list
    uint32_t pieces;            // of a row: dimensions over PIECE_DIMS, rounded up
    uint32_t stages, b_bufs;
    uint32_t raw_pitch;         // RaBitQ: bytes between rows of sign bits in shared memory
    uint32_t kchunks;           // SQ8: 16-byte cores per row of the tiled copy
    const int8_t* codes_t;      // SQ8: the tiled copy
    const unsigned char* terms; // [nq][B_TERMS][pieces * 128 bytes] the queries' operand rows
    const float* qscale;        // [nq] of the int8 terms
    const int32_t* qsum;        // RaBitQ: [nq][4] sums of the three terms
    const float* row_norm;      // |x|^2 by position (L2 over fp32 / bf16 / fp16 rows; the score leaves |q|^2 out);
                                // RaBitQ: pairs |x|^2, -2 |x| / error
    const uint32_t* pos_mask;   // bit by position: the id filter rejects the row; or null
    uint32_t l2;
    uint32_t spin_limit;
    int* error_flag;
};

// ---- grouping the pairs by list -------------------------------------------------------------
// pairs_prepare_kernel counted the pairs of every list and gave each its rank; one CTA turns the counts into
// places and the number of items, a grid scatters pairs and items.
struct TileGroup {
    uint32_t* count;          // [nlist] pairs per list (cleared here for the next batch)
    const uint32_t* rank;     // [pairs]
    const int32_t* probes;    // [pairs]
    uint32_t pairs, nlist, qt;
    uint32_t segment;         // rows of an item at most (a multiple of 8)
    const uint32_t* order;    // [nlist] lists, longest first: items that finish last are short
    const uint32_t* list_off;
    uint32_t* pair_off;       // [nlist]
    uint32_t* item_off;       // [nlist]
    uint32_t* list_pairs;     // [nlist] the counts, kept
    uint32_t* queue;          // [0] number of items, [1] cleared
    TilePair* tile_pairs;
    TileItem* items;
    uint32_t nprobe;
    PairTable t;
    const uint32_t* group_off; // SQ8 or null
};

__global__ void __launch_bounds__(1024)
tile_places_kernel(const TileGroup g) {
    __shared__ uint32_t part[32];
    __shared__ uint32_t carry[2];
    if (threadIdx.x < 2) {
        carry[threadIdx.x] = 0;
    }
    constexpr uint32_t PER = 4;
    for (uint32_t l0 = 0; l0 < g.nlist; l0 += 1024 * PER) {
        uint32_t list[PER], cnt[PER], its[PER], sum = 0, tiles = 0;
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) {
            const uint32_t i = l0 + threadIdx.x * PER + j;
            list[j] = i < g.nlist ? __ldg(g.order + i) : 0xFFFFFFFFu;
        }
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) {
            cnt[j] = list[j] != 0xFFFFFFFFu ? g.count[list[j]] : 0u;
            its[j] = cnt[j] > 0 ? (cnt[j] + g.qt - 1) / g.qt *
                                      ((__ldg(g.list_off + list[j] + 1) - __ldg(g.list_off + list[j]) + g.segment - 1) / g.segment)
                                : 0u;
            sum += cnt[j];
            tiles += its[j];
        }
        const uint32_t sum_incl = block_inclusive_sum<1024>(sum, part);
        const uint32_t tile_incl = block_inclusive_sum<1024>(tiles, part);
        uint32_t at = carry[0] + sum_incl - sum, tat = carry[1] + tile_incl - tiles;
        __syncthreads();
        if (threadIdx.x == 1023) {
            carry[0] += sum_incl;
            carry[1] += tile_incl;
        }
#pragma unroll
        for (uint32_t j = 0; j < PER; ++j) {
            if (list[j] != 0xFFFFFFFFu) {
                g.pair_off[list[j]] = at;
                g.item_off[list[j]] = tat;
                g.list_pairs[list[j]] = cnt[j];
                g.count[list[j]] = 0;
                at += cnt[j];
                tat += its[j];
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        g.queue[0] = carry[1];
        g.queue[1] = 0;
    }
}

__global__ void __launch_bounds__(256)
tile_scatter_kernel(const TileGroup g) {
    const uint32_t e = blockIdx.x * 256 + threadIdx.x;
    if (e < g.pairs) {
        const int32_t l = __ldg(g.probes + e);
        const uint32_t r = __ldg(g.rank + e);
        if (r != 0xFFFFFFFFu) {
            const uint32_t q = e / g.nprobe;
            g.tile_pairs[__ldg(g.pair_off + l) + r] = TilePair{q, 0u, q * g.t.stride + __ldg(g.t.base + e)};
        }
    }
    if (e < g.nlist) {
        const uint32_t n = g.list_pairs[e];
        TileItem* dst = g.items + g.item_off[e];
        const uint32_t p0 = g.pair_off[e];
        const uint32_t lbeg = __ldg(g.list_off + e);
        const uint32_t len = n > 0 ? __ldg(g.list_off + e + 1) - lbeg : 0u;
        const uint32_t goff = g.group_off != nullptr ? __ldg(g.group_off + e) : 0u;
        for (uint32_t row0 = 0; row0 < len; row0 += g.segment) {
            for (uint32_t i = 0; i * g.qt < n; ++i) {
                *dst++ = TileItem{lbeg + row0, min(len - row0, g.segment), p0 + i * g.qt, min(g.qt, n - i * g.qt), row0, goff + row0 / 8, 0u, 0u};
            }
        }
    }
}

// ---- SQ8 lists that a few queries probe ----------------------------------------------------
// pair_scan_kernel reads a list's rows once for every query, and what bounds it is that traffic from L2 (100 queries of 640
// dimensions, three per list: 1 GB, 144 us).  With two to four queries per list, too few for tensor-core tiles, the pairs are grouped by
// list all the same and a CTA streams up to SHARED_SEGMENT rows of a list past up to SHARED_QUERIES of them: 99 us, 111 with the grouping.
constexpr int SHARED_QUERIES = 4;
constexpr uint32_t SHARED_SEGMENT = 256;

template <bool L2>
__global__ void __launch_bounds__(RS_ROWS)
shared_scan_kernel(const PairScan p, const TileItem* __restrict__ items, uint32_t* __restrict__ queue, const TilePair* __restrict__ pairs) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_item;
    unsigned char* const terms = smem + RS_STAGES * RS_STAGE;
    const uint32_t n_items = queue[0], per_query = 3 * p.qstride;
    for (;;) {
        __syncthreads();   // (the item before is done with the queries)
        if (threadIdx.x == 0) {
            s_item = atomicAdd(queue + 1, 1u);
        }
        __syncthreads();
        if (s_item >= n_items) {
            return;
        }
        const uint4 head = __ldg(reinterpret_cast<const uint4*>(items + s_item));
        const uint32_t lbeg = head.x, len = head.y, pair0 = head.z, live = head.w, row0 = __ldg(&items[s_item].row0);
        float qa[SHARED_QUERIES], cq[SHARED_QUERIES];
        uint32_t* out[SHARED_QUERIES];
#pragma unroll
        for (int j = 0; j < SHARED_QUERIES; ++j) {
            if (static_cast<uint32_t>(j) < live) {
                const TilePair pair = pairs[pair0 + j];
                qa[j] = __ldg(p.s.qa + pair.q);
                cq[j] = p.s.coef_c * __ldg(p.qscale + pair.q);
                out[j] = reinterpret_cast<uint32_t*>(p.t.scores) + pair.out + row0;
                const uint4* src = reinterpret_cast<const uint4*>(p.qw8 + static_cast<uint64_t>(pair.q) * per_query);
                for (uint32_t i = threadIdx.x; i < per_query / 16; i += RS_ROWS) {
                    reinterpret_cast<uint4*>(terms + j * per_query)[i] = __ldg(src + i);
                }
            } else {
                qa[j] = cq[j] = 0.f;
                out[j] = nullptr;
            }
        }
        RowAcc<ROW_SQ8, L2, SHARED_QUERIES> acc;
        acc.live = live;
        row_stream<16>(p.s.codes + static_cast<uint64_t>(lbeg) * p.s.code_stride, p.s.code_stride, p.row_bytes, p.s.dim, len, 0, 1, smem,
                       reinterpret_cast<const float*>(terms), p.qstride, acc, [&](uint64_t row, bool valid) {
                           if (!valid) {
                               return;
                           }
                           const uint32_t pos = lbeg + static_cast<uint32_t>(row);
                           const float norm = p.s.coef_b * __ldg(p.s.code_norm + pos);
                           const bool filtered = p.s.filter_pos_inner != nullptr && scan_row_filtered(p.s, pos);
#pragma unroll
                           for (int j = 0; j < SHARED_QUERIES; ++j) {
                               if (static_cast<uint32_t>(j) < live) {
                                   const float f = sq8_term_sum(acc.a1[j], acc.a2[j], acc.a3[j], p.s.dim <= SQ8_NARROW_DIMS);
                                   out[j][row] = filtered ? SCORE_FILTERED : __float_as_uint(fmaf(cq[j], f, norm) + qa[j]);
                               }
                           }
                       });
    }
}

// ---- the kernel -----------------------------------------------------------------------------
struct TileShared {
    uint64_t full[TILE_MAX_STAGES], freed[TILE_MAX_STAGES];   // operand stages
    uint64_t raw_full[TILE_MAX_STAGES], raw_free[2];          // rows as they are stored, before conversion
    uint64_t desc_full[TILE_DESCS], desc_free[TILE_DESCS];
    uint64_t item_full[2], item_free[2];                      // B operand and constants of an item
    uint64_t b_free[2];
    uint64_t acc_full[2], acc_free[2];
    uint32_t tmem_base, failed;
    TileItem desc[TILE_DESCS];
    // two items deep: where the scores of the item's queries go and their constants
    alignas(16) uint64_t out[2][64];
    float c0[2][64], c1[2][64];
    int32_t t1[2][64], t2[2][64], t3[2][64];
};

// Two bf16 terms of eight values: x = hi + lo.
__device__ __forceinline__ void
split_bf16x8(const float (&x)[8], uint4& hi, uint4& lo) {
    uint32_t h[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float a = x[2 * i], b = x[2 * i + 1];
        uint32_t w;
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(b), "f"(a));
        h[i] = w;
        const float ra = a - __uint_as_float(w << 16), rb = b - __uint_as_float(w & 0xFFFF0000u);
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(w) : "f"(rb), "f"(ra));
        l[i] = w;
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

// fp32 rows (16-byte aligned) -> [rows][2][pitch] bf16 terms, zero past dim; pitch = dim rounded up to 8.  A thread per eight dimensions.
__global__ void __launch_bounds__(256)
split_rows_kernel(const uint8_t* __restrict__ rows, uint64_t n, uint32_t dim, uint32_t stride, uint32_t pitch, uint16_t* __restrict__ out) {
    const uint64_t e = static_cast<uint64_t>(blockIdx.x) * 256 + threadIdx.x;
    const uint32_t units = pitch / 8;
    const uint64_t r = e / units;
    if (r >= n) {
        return;
    }
    const uint32_t d0 = static_cast<uint32_t>(e - r * units) * 8;
    const float* src = reinterpret_cast<const float*>(rows + r * stride);
    float x[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; i += 4) {
        if (d0 + i + 4 <= dim) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(src + d0 + i));
            x[i] = v.x;
            x[i + 1] = v.y;
            x[i + 2] = v.z;
            x[i + 3] = v.w;
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                x[i + j] = d0 + i + j < dim ? __ldg(src + d0 + i + j) : 0.f;
            }
        }
    }
    uint4 hi, lo;
    split_bf16x8(x, hi, lo);
    uint16_t* to = out + r * 2 * pitch + d0;
    *reinterpret_cast<uint4*>(to) = hi;
    *reinterpret_cast<uint4*>(to + pitch) = lo;
}

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: 8-row groups of 1 KiB; a k-step of 32 bytes is two
// 16-byte units further into the line.
__device__ __forceinline__ uint64_t
umma_desc_sw128(uint32_t smem_addr) {
    return static_cast<uint64_t>((smem_addr >> 4) & 0x3FFFu) | (1ull << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) |
           (2ull << 61);
}

// Where unit kc (16 bytes) of row r sits in a [rows x 128 bytes] swizzled block.
__device__ __forceinline__ uint32_t
swizzled(uint32_t r, uint32_t kc) {
    return r * 128 + ((kc ^ (r & 7u)) << 4);
}

// One box of a tiled tensor map -> shared memory, completion counted in bytes on `bar`.
__device__ __forceinline__ void
tma_load_2d(void* dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void
tma_load_3d(void* dst, const CUtensorMap* map, uint32_t x, uint32_t y, uint32_t z, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

// 8 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void
tmem_load_8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

// Smallest of the warp's fp32 bit patterns; NaNs do not take part (all NaN: NaN).
__device__ __forceinline__ float
warp_min_f32(uint32_t bits) {
    float out;
    asm("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(out) : "f"(__uint_as_float(bits)));
    return out;
}

// A warp's wait: one lane polls (32 lanes polling one barrier are 32 operations on it, and eight warps of them kept
// the L1 pipe 97 % busy), the others wait for it.
__device__ __forceinline__ bool
tile_wait(uint64_t* bar, uint32_t parity, const volatile uint32_t* failed, uint32_t limit, uint32_t lane) {
    bool ok = true;
    if (lane == 0) {
        ok = tcs_wait(bar, parity, failed, limit);
    }
    ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
    __syncwarp();
    return ok;
}

// A warp's part of an operand is written: visible to the MMAs (async proxy), one arrival per warp.
__device__ __forceinline__ void
tile_publish(uint64_t* bar, uint32_t lane) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncwarp();
    if (lane == 0) {
        mbar_arrive(bar);
    }
}

// kind::f16 (fp16 or bf16 operands) and kind::i8 instruction descriptors, M 128.
template <int FMT>
__device__ __forceinline__ uint32_t
tile_idesc(uint32_t n) {
    if (TileFmt<FMT>::INT8) {
        return umma_idesc_s8(128, n);
    }
    return FMT == ROW_FP16 ? umma_idesc_f16(128, n) : umma_idesc_bf16(128, n);
}

// QT queries per item at most (16, 32 or 64).
template <int FMT, int QT>
__global__ void __launch_bounds__(TileFmt<FMT>::THREADS, 1)
tile_scan_kernel(const __grid_constant__ TileScan p) {
    using F = TileFmt<FMT>;
    constexpr uint32_t STAGE = F::STAGE;
    constexpr uint32_t B_PIECE = F::B_TERMS * QT * TILE_PIECE;
    constexpr uint32_t COL_STEP = F::EPI / 4 * 8;   // columns that the warps of 32 rows drain at a time
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ TileShared sh;
    // the swizzle permutes by address bits: blocks start on 1 KiB
    unsigned char* const smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const uint32_t stages = p.stages, pieces = p.pieces, dim = p.s.dim;
    unsigned char* const b_smem = smem + stages * STAGE;
    const uint32_t b_bytes = pieces * B_PIECE;
    unsigned char* const raw_smem = b_smem + p.b_bufs * b_bytes;
    const volatile uint32_t* failed = &sh.failed;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < stages; ++s) {
            mbar_init(&sh.full[s], F::CONVERT ? TILE_CONV_WARPS : 1);
            mbar_init(&sh.freed[s], 1);
            mbar_init(&sh.raw_full[s], 1);
        }
        for (uint32_t i = 0; i < TILE_DESCS; ++i) {
            mbar_init(&sh.desc_full[i], 1);
            mbar_init(&sh.desc_free[i], F::EPI + 1 + TILE_QUERY_WARPS + (F::CONVERT ? TILE_CONV_WARPS : 0));
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.raw_free[i], TILE_CONV_WARPS);
            mbar_init(&sh.item_full[i], TILE_QUERY_WARPS);
            mbar_init(&sh.item_free[i], F::EPI);
            mbar_init(&sh.b_free[i], 1);
            mbar_init(&sh.acc_full[i], 1);
            mbar_init(&sh.acc_free[i], F::EPI);
        }
        sh.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == F::EPI) {
        tmem_alloc(&sh.tmem_base, 2 * TILE_ACC_COLS);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = sh.tmem_base;
    bool ok = true;
    // The item number n of this CTA; false at the end of the queue or when another role has failed.
    auto next_item = [&](uint32_t n, TileItem& it) -> bool {
        const uint32_t slot = n % TILE_DESCS;
        ok = tile_wait(&sh.desc_full[slot], (n / TILE_DESCS) & 1u, failed, p.spin_limit, lane);
        if (!ok) {
            return false;
        }
        it = sh.desc[slot];
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&sh.desc_free[slot]);
        }
        return it.len != 0;
    };

    if (warp == F::EPI + 1) {
        // ---------------- the work queue and the copies of rows ----------------
        const uint32_t n_items = p.queue[0];
        uint32_t stage = 0, phase = 0, filled = 0, raw = 0;
        auto fetch = [&](uint32_t i) -> TileItem {
            TileItem it{};
            if (i < n_items) {
                const uint4* src = reinterpret_cast<const uint4*>(p.items + i);
                const uint4 a = __ldg(src), b = __ldg(src + 1);
                it = TileItem{a.x, a.y, a.z, a.w, b.x, b.y, 0u, 0u};
            }
            return it;
        };
        auto ticket = [&]() -> uint32_t {   // (the same number for all lanes)
            uint32_t t = 0;
            if (lane == 0) {
                t = atomicAdd(p.queue + 1, 1u);
            }
            return t;
        };
        // the next item's description and the ticket after it are under way while an item's rows are copied
        TileItem next = fetch(__shfl_sync(0xffffffffu, ticket(), 0));
        uint32_t after = ticket();
        for (uint32_t n = 0;; ++n) {
            const uint32_t slot = n % TILE_DESCS;
            if (n >= TILE_DESCS) {
                ok = tile_wait(&sh.desc_free[slot], (n / TILE_DESCS - 1u) & 1u, failed, p.spin_limit, lane);
                if (!ok) {
                    break;
                }
            }
            const TileItem it = next;
            if (lane == 0) {
                sh.desc[slot] = it;
                mbar_arrive(&sh.desc_full[slot]);
            }
            if (it.len == 0) {
                break;
            }
            next = fetch(__shfl_sync(0xffffffffu, after, 0));
            after = ticket();
            for (uint32_t r0 = 0; r0 < it.len && ok; r0 += 128) {
                if (FMT == ROW_RABITQ) {
                    // the sign bits of 128 rows at once
                    const uint32_t buf = raw & 1u;
                    if (raw >= 2) {
                        ok = tile_wait(&sh.raw_free[buf], (raw / 2 - 1u) & 1u, failed, p.spin_limit, lane);
                    }
                    if (ok && lane == 0) {
                        mbar_expect_tx(&sh.raw_full[buf], 128 * p.raw_pitch);
                        tma_load_2d(raw_smem + buf * 128 * p.raw_pitch, &p.map, 0, it.lbeg + r0, &sh.raw_full[buf]);
                    }
                    ++raw;
                    continue;
                }
                for (uint32_t piece = 0; piece < pieces; ++piece) {
                    if (filled >= stages) {
                        ok = tile_wait(&sh.freed[stage], phase ^ 1u, failed, p.spin_limit, lane);
                        if (!ok) {
                            break;
                        }
                    }
                    unsigned char* dst = smem + stage * STAGE;
                    if (FMT == ROW_SQ8) {
                        // the tiled signed copy: of every 8-row group its cores of this piece, 16 groups
                        const uint32_t cores = min(8u, p.kchunks - piece * 8);
                        if (lane == 0) {
                            mbar_expect_tx(&sh.full[stage], 16 * cores * 128);
                        }
                        __syncwarp();
                        if (lane < 16) {
                            const int8_t* src = p.codes_t + (static_cast<uint64_t>(it.goff + r0 / 8 + lane) * p.kchunks + piece * 8) * 128;
                            bulk_copy_g2s(dst + lane * 1024, src, cores * 128, &sh.full[stage]);
                        }
                    } else if (lane == 0) {
                        uint64_t* bar = F::CONVERT ? &sh.raw_full[stage] : &sh.full[stage];
                        mbar_expect_tx(bar, STAGE);
                        if (FMT == ROW_F32_SPLIT) {
                            tma_load_3d(dst, &p.map, piece * 64, 0, it.lbeg + r0, bar);
                            tma_load_3d(dst + TILE_A_TERM, &p.map, piece * 64, 1, it.lbeg + r0, bar);
                        } else if (FMT == ROW_F32) {
                            tma_load_2d(dst, &p.map, piece * 64, it.lbeg + r0, bar);
                            tma_load_2d(dst + TILE_A_TERM, &p.map, piece * 64 + 32, it.lbeg + r0, bar);
                        } else {
                            tma_load_2d(dst, &p.map, piece * 64, it.lbeg + r0, bar);
                        }
                    }
                    ++filled;
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
            }
            if (!ok) {
                break;
            }
        }
    } else if (warp == F::EPI) {
        // ---------------- MMA issue (one thread) ----------------
        if (elect_one()) {
            const uint64_t a0 = FMT == ROW_SQ8 ? umma_desc(smem_u32(smem), 128, 1024) : umma_desc_sw128(smem_u32(smem));
            const uint64_t b0 = umma_desc_sw128(smem_u32(b_smem));
            constexpr uint32_t A_STEP = FMT == ROW_SQ8 ? 16 : 2;   // descriptor units per k-step of 32 bytes
            // k-steps of the last piece: the rest of the row (fp32: a step holds eight of the first 32 dimensions)
            const uint32_t rest = dim - (pieces - 1) * F::PIECE_DIMS;
            const uint32_t last_steps = FMT == ROW_F32 ? min(4u, (rest + 7) / 8) : (rest + F::PIECE_DIMS / 4 - 1) / (F::PIECE_DIMS / 4);
            uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0, tiles = 0;
            for (uint32_t n = 0; ok; ++n) {
                const uint32_t slot = n % TILE_DESCS;
                ok = tcs_wait(&sh.desc_full[slot], (n / TILE_DESCS) & 1u, failed, p.spin_limit);
                if (!ok) {
                    break;
                }
                const uint32_t len = sh.desc[slot].len, nqt = sh.desc[slot].nqt;
                mbar_arrive(&sh.desc_free[slot]);
                if (len == 0) {
                    break;
                }
                const uint32_t qn = (nqt + 15) & ~15u;
                const uint32_t idesc = tile_idesc<FMT>(F::B_TERMS * qn), idesc_lo = tile_idesc<FMT>(qn);
                const uint32_t buf = p.b_bufs == 2 ? n & 1u : 0u;
                ok = tcs_wait(&sh.item_full[n & 1u], (n >> 1) & 1u, failed, p.spin_limit);
                for (uint32_t r0 = 0; r0 < len && ok; r0 += 128) {
                    if (tiles >= 2) {
                        ok = tcs_wait(&sh.acc_free[acc], acc_phase ^ 1u, failed, p.spin_limit);
                        if (!ok) {
                            break;
                        }
                    }
                    const uint32_t d_tmem = tmem_base + acc * TILE_ACC_COLS;
                    for (uint32_t piece = 0; piece < pieces; ++piece) {
                        ok = tcs_wait(&sh.full[stage], phase, failed, p.spin_limit);
                        if (!ok) {
                            break;
                        }
                        tc_fence_after_sync();
                        const uint64_t a = a0 + (stage * STAGE >> 4);
                        const uint64_t b = b0 + ((buf * b_bytes + piece * B_PIECE) >> 4);
                        const uint32_t steps = piece + 1 == pieces ? last_steps : 4u;
                        for (uint32_t ks = 0; ks < steps; ++ks) {
                            const uint32_t accumulate = (piece | ks) != 0 ? 1u : 0u;
                            if (F::INT8) {
                                umma_s8(d_tmem, a + ks * A_STEP, b + ks * 2, idesc, accumulate);
                            } else {
                                umma_bf16(d_tmem, a + ks * A_STEP, b + ks * 2, idesc, accumulate);
                            }
                            if (F::SPLIT) {   // lo terms of the rows against hi terms of the queries
                                umma_bf16(d_tmem, a + (TILE_A_TERM >> 4) + ks * A_STEP, b + ks * 2, idesc_lo, 1u);
                            }
                        }
                        umma_commit(&sh.freed[stage]);
                        if (piece + 1 == pieces) {
                            umma_commit(&sh.acc_full[acc]);
                            if (r0 + 128 >= len) {
                                umma_commit(&sh.b_free[buf]);
                            }
                        }
                        if (++stage == stages) {
                            stage = 0;
                            phase ^= 1u;
                        }
                    }
                    ++tiles;
                    if (++acc == 2) {
                        acc = 0;
                        acc_phase ^= 1u;
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp > F::EPI + 1 && warp < F::EPI + 2 + TILE_QUERY_WARPS) {
        // ---------------- an item ahead: the queries' terms (B) and constants ----------------
        // Query j belongs to warp j % 4 of the role, lane j / 4 of it: no warp waits for another.
        const uint32_t qwarp = warp - (F::EPI + 2);
        const uint32_t j = lane * TILE_QUERY_WARPS + qwarp;
        TileItem it;
        for (uint32_t n = 0; next_item(n, it); ++n) {
            const uint32_t slot = n & 1u, buf = p.b_bufs == 2 ? slot : 0u;
            // (while the waits run, the pairs are on their way)
            uint32_t q = 0;
            uint64_t out = 0;
            if (j < it.nqt) {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(p.pairs + it.pair0 + j));
                q = v.x;
                out = (static_cast<uint64_t>(v.z) | (static_cast<uint64_t>(v.w) << 32)) + it.row0;
            }
            if (n >= 2) {
                ok = tile_wait(&sh.item_free[slot], ((n >> 1) - 1u) & 1u, failed, p.spin_limit, lane);
            }
            if (ok && n >= p.b_bufs) {
                ok = tile_wait(&sh.b_free[buf], (n / p.b_bufs - 1u) & 1u, failed, p.spin_limit, lane);
            }
            if (!ok) {
                break;
            }
            unsigned char* bd = b_smem + buf * b_bytes;
            const uint32_t per_row = pieces * 8;             // 16-byte units of a term
            const uint32_t qn = (it.nqt + 15) & ~15u;
            // (the rows of queries past the item's are left as they are: their columns are not read)
            for (uint32_t i = 0; i * TILE_QUERY_WARPS + qwarp < it.nqt; ++i) {
                const uint64_t qq = __shfl_sync(0xffffffffu, q, i);
                const uint32_t qi = i * TILE_QUERY_WARPS + qwarp;
                const unsigned char* src = p.terms + qq * F::B_TERMS * per_row * 16;
                for (uint32_t u = lane; u < F::B_TERMS * per_row; u += 32) {
                    const uint32_t term = u / per_row, k = u - term * per_row;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                     smem_u32(bd + (k >> 3) * B_PIECE + swizzled(term * qn + qi, k & 7u))),
                                 "l"(src + u * 16)
                                 : "memory");
                }
            }
            if (j < it.nqt) {
                sh.out[slot][j] = out;
                if (FMT == ROW_SQ8) {
                    sh.c0[slot][j] = __ldg(p.s.qa + q);
                    sh.c1[slot][j] = p.s.coef_c * __ldg(p.qscale + q);
                } else if (FMT == ROW_RABITQ) {
                    sh.c0[slot][j] = __ldg(p.s.queries + static_cast<uint64_t>(q) * (dim + 1) + dim);
                    sh.c1[slot][j] = __ldg(p.qscale + q);
                    const int4 t = __ldg(reinterpret_cast<const int4*>(p.qsum) + q);
                    sh.t1[slot][j] = t.x;
                    sh.t2[slot][j] = t.y;
                    sh.t3[slot][j] = t.z;
                }
            }
            asm volatile("cp.async.wait_all;" ::: "memory");
            tile_publish(&sh.item_full[slot], lane);
        }
    } else if (F::CONVERT && warp >= F::EPI + 2 + TILE_QUERY_WARPS) {
        // ---------------- stored rows -> operands, in shared memory ----------------
        const uint32_t cwarp = warp - (F::EPI + 2 + TILE_QUERY_WARPS);
        constexpr uint32_t ROWS = 128 / TILE_CONV_WARPS;     // of every tile, for a warp
        const uint32_t kc = lane & 7u, rr = cwarp * ROWS + (lane >> 3);   // eight lanes per row, four rows at a time
        uint32_t stage = 0, phase = 0, filled = 0, raw = 0;
        TileItem it;
        for (uint32_t n = 0; ok && next_item(n, it); ++n) {
            for (uint32_t r0 = 0; r0 < it.len && ok; r0 += 128) {
                const unsigned char* bits = raw_smem + (raw & 1u) * 128 * p.raw_pitch;
                if (FMT == ROW_RABITQ) {
                    ok = tile_wait(&sh.raw_full[raw & 1u], (raw >> 1) & 1u, failed, p.spin_limit, lane);
                }
                for (uint32_t piece = 0; piece < pieces && ok; ++piece) {
                    unsigned char* dst = smem + stage * STAGE;
                    if (FMT == ROW_RABITQ) {
                        if (filled >= stages) {
                            ok = tile_wait(&sh.freed[stage], phase ^ 1u, failed, p.spin_limit, lane);
                        }
                        if (!ok) {
                            break;
                        }
                        // bits s, s + 8, s + 16, s + 24 of a word become the four bytes of one: two instructions per
                        // four dimensions (the queries' terms are in the same order, see rabitq_query_kernel)
                        uint32_t w[ROWS / 4];
#pragma unroll
                        for (uint32_t j = 0; j < ROWS / 4; ++j) {
                            w[j] = *reinterpret_cast<const uint32_t*>(bits + (rr + j * 4) * p.raw_pitch + piece * 16 + (kc >> 1) * 4) >> ((kc & 1u) * 4);
                        }
#pragma unroll
                        for (uint32_t j = 0; j < ROWS / 4; ++j) {
                            constexpr uint32_t ONES = 0x01010101u;
                            *reinterpret_cast<uint4*>(dst + swizzled(rr + j * 4, kc)) =
                                make_uint4(w[j] & ONES, (w[j] >> 1) & ONES, (w[j] >> 2) & ONES, (w[j] >> 3) & ONES);
                        }
                    } else {
                        // fp32, in place: dimensions 0-31 of the piece lie in the first block and 32-63 in the second,
                        // 128 bytes of either per row; the hi terms take the row's line of the first, the lo terms of
                        // the second.  Unit kc holds dimensions 4 kc .. + 3 and 32 + 4 kc .. + 3 (the queries' terms too).
                        ok = tile_wait(&sh.raw_full[stage], phase, failed, p.spin_limit, lane);
                        if (!ok) {
                            break;
                        }
                        uint4 a[ROWS / 4], b[ROWS / 4];
#pragma unroll
                        for (uint32_t j = 0; j < ROWS / 4; ++j) {
                            const unsigned char* src = dst + (rr + j * 4) * 128 + kc * 16;
                            a[j] = *reinterpret_cast<const uint4*>(src);
                            b[j] = *reinterpret_cast<const uint4*>(src + TILE_A_TERM);
                        }
                        __syncwarp();
#pragma unroll
                        for (uint32_t j = 0; j < ROWS / 4; ++j) {
                            const float x[8] = {__uint_as_float(a[j].x), __uint_as_float(a[j].y), __uint_as_float(a[j].z), __uint_as_float(a[j].w),
                                                __uint_as_float(b[j].x), __uint_as_float(b[j].y), __uint_as_float(b[j].z), __uint_as_float(b[j].w)};
                            uint4 hi, lo;
                            split_bf16x8(x, hi, lo);
                            *reinterpret_cast<uint4*>(dst + swizzled(rr + j * 4, kc)) = hi;
                            *reinterpret_cast<uint4*>(dst + TILE_A_TERM + swizzled(rr + j * 4, kc)) = lo;
                        }
                    }
                    tile_publish(&sh.full[stage], lane);
                    ++filled;
                    if (++stage == stages) {
                        stage = 0;
                        phase ^= 1u;
                    }
                }
                if (FMT == ROW_RABITQ) {
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&sh.raw_free[raw & 1u]);
                    }
                    ++raw;
                }
            }
        }
    } else if (warp < F::EPI) {
        // ---------------- epilogue: one thread per row of the tile, the warps of 32 rows share the queries ----------------
        const uint32_t quarter = warp & 3u, share = warp >> 2;
        const uint32_t row = quarter * 32 + lane;
        uint32_t tile = 0;
        TileItem it;
        for (uint32_t n = 0; ok && next_item(n, it); ++n) {
            const uint32_t slot = n & 1u;
            const uint32_t qn = (it.nqt + 15) & ~15u;
            // what a row contributes to its scores, one tile ahead: whether it takes part, its norm terms
            struct RowPart {
                float x0, x1;
                bool drop;
            };
            auto row_part = [&](uint32_t r) -> RowPart {
                RowPart part{0.f, 0.f, true};
                if (r < it.len) {
                    const uint32_t pos = it.lbeg + r;
                    if (FMT == ROW_SQ8) {
                        part.x0 = p.s.coef_b * __ldg(p.row_norm + pos);
                    } else if (FMT == ROW_RABITQ) {
                        const float2 v = __ldg(reinterpret_cast<const float2*>(p.row_norm) + pos);
                        part.x0 = v.x;
                        part.x1 = v.y;
                    } else if (p.l2 != 0) {
                        part.x0 = __ldg(p.row_norm + pos);
                    }
                    part.drop = p.pos_mask != nullptr && ((__ldg(p.pos_mask + (pos >> 5)) >> (pos & 31u)) & 1u) != 0;
                }
                return part;
            };
            RowPart ahead = row_part(row);
            ok = tile_wait(&sh.item_full[slot], (n >> 1) & 1u, failed, p.spin_limit, lane);
            for (uint32_t r0 = 0; r0 < it.len && ok; r0 += 128, ++tile) {
                const uint32_t r = r0 + row, acc = tile & 1u;
                const RowPart part = ahead;
                if (r0 + 128 < it.len) {
                    ahead = row_part(r + 128);
                }
                const float x0 = part.x0, x1 = part.x1;
                ok = tile_wait(&sh.acc_full[acc], (tile >> 1) & 1u, failed, p.spin_limit, lane);
                if (!ok) {
                    break;
                }
                tc_fence_after_sync();
                const uint32_t taddr = tmem_base + ((quarter * 32u) << 16) + acc * TILE_ACC_COLS;
                if (r0 + quarter * 32 < it.len) {   // (the warp's rows are one group of 32 scores)
                    uint32_t* const scores = reinterpret_cast<uint32_t*>(p.t.scores) + r;
                    for (uint32_t g = share * 8; g < it.nqt; g += COL_STEP) {
                        uint32_t v1[8], v2[8], v3[8];
                        tmem_load_8(taddr + g, v1);
                        if (F::B_TERMS >= 2) {
                            tmem_load_8(taddr + qn + g, v2);
                        }
                        if (F::B_TERMS >= 3) {
                            tmem_load_8(taddr + 2 * qn + g, v3);
                        }
                        // destinations in wide reads, before the stores: a read between two of them would wait
                        ulonglong2 to[4];
#pragma unroll
                        for (uint32_t i = 0; i < 4; ++i) {
                            to[i] = *reinterpret_cast<const ulonglong2*>(&sh.out[slot][g + 2 * i]);
                        }
                        tmem_load_wait();
                        float least = 0.f;   // of column g + lane
#pragma unroll
                        for (uint32_t i = 0; i < 8; ++i) {
                            const uint32_t j = g + i;
                            float v;
                            if (FMT == ROW_SQ8) {
                                const float f = sq8_term_sum(static_cast<int32_t>(v1[i]), static_cast<int32_t>(v2[i]), static_cast<int32_t>(v3[i]),
                                                             dim <= SQ8_NARROW_DIMS);
                                v = fmaf(sh.c1[slot][j], f, x0) + sh.c0[slot][j];
                            } else if (FMT == ROW_RABITQ) {
                                // |x|^2 + |q|^2 - 2 |x| |q| (ip / error); the set bits' sum S gives ip = 2 S - (sum of all).  (Signed
                                // sums of terms up to 127: 254 u2 + u3 fits 32 bits to 66,000 dimensions, the row map ends at 1920.)
                                const int32_t u1 = 2 * static_cast<int32_t>(v1[i]) - sh.t1[slot][j];
                                const int32_t u2 = 2 * static_cast<int32_t>(v2[i]) - sh.t2[slot][j];
                                const int32_t u3 = 2 * static_cast<int32_t>(v3[i]) - sh.t3[slot][j];
                                const float f = fmaf(static_cast<float>(u2 * 254 + u3), 1.0f / 64516.0f, static_cast<float>(u1));
                                const float qn2 = sh.c0[slot][j];
                                v = fmaf(x1 * qn2, f * sh.c1[slot][j], fmaf(qn2, qn2, x0));
                            } else {
                                float ip = __uint_as_float(v1[i]);
                                if (F::SPLIT) {
                                    ip += __uint_as_float(v2[i]);
                                }
                                v = fmaf(p.l2 != 0 ? -2.0f : -1.0f, ip, x0);   // (a negated NaN would rank first)
                            }
                            const uint32_t bits = part.drop ? SCORE_FILTERED : __float_as_uint(v);
                            if (j < it.nqt) {
                                scores[(i & 1u) != 0 ? to[i >> 1].y : to[i >> 1].x] = bits;
                            }
                            const float low = warp_min_f32(bits);
                            least = lane == i ? low : least;
                        }
                        if (lane < 8 && g + lane < it.nqt) {
                            p.t.minima[(sh.out[slot][g + lane] + r0 + quarter * 32) >> 5] = ScoreSource<>::ordered(__float_as_uint(least));
                        }
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sh.acc_free[acc]);
                }
            }
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&sh.item_free[slot]);
            }
        }
    }
    if (!ok) {
        sh.failed = 1;
        atomicOr(p.error_flag, 1);
    }
    tc_fence_before_sync();
    __syncthreads();
    if (sh.failed != 0) {
        tc_drain_pause();   // a wait gave up: let the copies and MMAs still in flight land before the CTA lets go
        __syncthreads();
    }
    if (warp == F::EPI) {
        tmem_dealloc(tmem_base, 2 * TILE_ACC_COLS);
    }
}

}  // namespace vb200
