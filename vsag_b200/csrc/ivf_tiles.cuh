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
// The rows keep their stored form; the loader warps turn a piece of 128 bytes of operand per row into the layout
// the MMA descriptors describe on its way to shared memory.  That is the 128-byte swizzle -- a row's piece is one
// 128-byte line, its 16-byte units permuted by the row number -- because eight lanes can then read one line of a
// row and write one line of the operand: with unswizzled cores either the loads touch a line per lane or the stores
// hit the same banks, and the kernel spent 82 % of its cycles on those wavefronts (500 us instead of 280 for
// 1000 queries against 32 lists each of 500k x 128 fp32).  The codecs:
//   fp32        two bf16 terms x = hi + lo; hi*hi + lo*hi and hi*lo are accumulated (the dropped terms are below
//               2^-16 |x||q|)
//   bf16, fp16  the codes as they are; every product is exact in fp32
//   sq8         code - 128 as signed bytes against three int8 terms of the query's weights, exact int32 sums
//   rabitq      the sign bits as bytes 0 / 1 against three int8 terms of the query; sum over set bits = (sum of all
//               terms + signed sum) / 2
// Each loader thread holds its part of the next two or three pieces in registers while it converts the current one,
// across tiles and items, so 64 KB or more per SM are always in flight.
#pragma once

#include "ivf_pairs.cuh"
#include "ivf_scan_tc.cuh"

namespace vb200 {

constexpr int TILE_LOAD_WARPS = 8;
constexpr int TILE_LOADERS = 32 * TILE_LOAD_WARPS;
constexpr int TILE_EPI_WARPS = 8;
constexpr int TILE_THREADS = 32 * (TILE_EPI_WARPS + 1 + TILE_LOAD_WARPS);   // warps 0-7 epilogue, 8 MMA, then the loaders
constexpr uint32_t TILE_PIECE = 128;                        // operand bytes per row and piece
constexpr uint32_t TILE_A_TERM = 128 * TILE_PIECE;          // 16 KiB
constexpr uint32_t TILE_MAX_STAGES = 6;
constexpr uint32_t TILE_ACC_COLS = 256;                     // tensor-memory columns per accumulator, two of them

// How a codec becomes MMA operands.
template <int FMT>
struct TileFmt {
    static constexpr bool INT8 = FMT == ROW_SQ8 || FMT == ROW_RABITQ;
    static constexpr uint32_t A_TERMS = FMT == ROW_F32 ? 2 : 1;
    static constexpr uint32_t B_TERMS = INT8 ? 3 : (FMT == ROW_F32 ? 2 : 1);
    static constexpr uint32_t PIECE_DIMS = INT8 ? 128 : 64;
};

// Lists of very different lengths are the rule (a list that many queries probe is often a long one): an item is at
// most TILE_SEGMENT rows of a list, so that no CTA is left with one long list at the end.
constexpr uint32_t TILE_SEGMENT = 1024;

struct TileItem {
    uint32_t list, pair0, nqt, row0;   // rows row0 .. row0 + TILE_SEGMENT of the list
};

struct TileScan {
    ScanParams s;               // rows, list_off, filter, constants; queries (RaBitQ: processed)
    PairTable t;
    uint32_t nprobe;
    const TileItem* items;
    const uint32_t* n_items;    // [1]
    const uint32_t* pair_ids;   // pairs (query * nprobe + rank) grouped by list
    uint32_t pieces;            // of a row: dimensions over PIECE_DIMS, rounded up
    uint32_t stages, b_bufs;
    uint32_t qstride;           // int8 terms: bytes per term
    const int8_t* qw8;          // [nq][3][qstride]
    const float* qscale;        // [nq]
    const int32_t* qsum;        // RaBitQ: [nq][4] sums of the three terms
    const float* row_norm;      // L2 over fp32 / bf16 / fp16 rows: |x|^2 by position (the score leaves |q|^2 out)
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
    const uint32_t* order;    // [nlist] lists, longest first: items that finish last are short
    const uint32_t* list_off;
    uint32_t* pair_off;       // [nlist]
    uint32_t* item_off;       // [nlist]
    uint32_t* list_pairs;     // [nlist] the counts, kept
    uint32_t* n_items;
    uint32_t* pair_ids;
    TileItem* items;
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
                                      ((__ldg(g.list_off + list[j] + 1) - __ldg(g.list_off + list[j]) + TILE_SEGMENT - 1) / TILE_SEGMENT)
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
        *g.n_items = carry[1];
    }
}

__global__ void __launch_bounds__(256)
tile_scatter_kernel(const TileGroup g) {
    const uint32_t e = blockIdx.x * 256 + threadIdx.x;
    if (e < g.pairs) {
        const int32_t l = __ldg(g.probes + e);
        const uint32_t r = __ldg(g.rank + e);
        if (r != 0xFFFFFFFFu) {
            g.pair_ids[__ldg(g.pair_off + l) + r] = e;
        }
    }
    if (e < g.nlist) {
        const uint32_t n = g.list_pairs[e];
        TileItem* dst = g.items + g.item_off[e];
        const uint32_t p0 = g.pair_off[e];
        const uint32_t len = n > 0 ? __ldg(g.list_off + e + 1) - __ldg(g.list_off + e) : 0u;
        for (uint32_t row0 = 0; row0 < len; row0 += TILE_SEGMENT) {
            for (uint32_t i = 0; i * g.qt < n; ++i) {
                *dst++ = TileItem{e, p0 + i * g.qt, min(g.qt, n - i * g.qt), row0};
            }
        }
    }
}

// ---- the kernel -----------------------------------------------------------------------------
struct TileShared {
    uint64_t full[TILE_MAX_STAGES], freed[TILE_MAX_STAGES];
    uint64_t b_full[2], b_free[2];
    uint64_t acc_full[2], acc_free[2];
    uint32_t tmem_base, failed;
    // where the running item's scores go and its queries' constants: a copy per epilogue warp, which therefore never
    // wait for one another
    uint64_t out[TILE_EPI_WARPS][64];
    float c0[TILE_EPI_WARPS][64], c1[TILE_EPI_WARPS][64];
    int32_t t1[TILE_EPI_WARPS][64], t2[TILE_EPI_WARPS][64], t3[TILE_EPI_WARPS][64];
};

// Instruction descriptor of kind::f16 with fp16 operands (bf16: umma_idesc_bf16).
__host__ __device__ constexpr uint32_t
umma_idesc_f16(uint32_t m, uint32_t n) {
    return (1u << 4) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

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

// 16 sign bits -> 16 bytes of 0 / 1.
__device__ __forceinline__ uint4
spread_bits16(uint32_t b) {
    auto four = [](uint32_t n) { return (n * 0x00204081u) & 0x01010101u; };
    return make_uint4(four(b & 15u), four((b >> 4) & 15u), four((b >> 8) & 15u), four((b >> 12) & 15u));
}

// One 16-byte operand unit per A term of row `row` (a code record), k-core `kc` of piece `piece`.
template <int FMT>
struct TileUnit {
    uint4 raw[FMT == ROW_F32 ? 2 : 1];
    uint2 bits;   // RaBitQ
    __device__ __forceinline__ void
    load(const uint8_t* row, bool valid, uint32_t piece, uint32_t kc, uint32_t dim) {
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        if (FMT == ROW_F32) {
            const uint32_t d0 = piece * 64 + kc * 8;
            const uint4* src = reinterpret_cast<const uint4*>(row + static_cast<size_t>(d0) * 4);
            raw[0] = valid && d0 < dim ? __ldg(src) : zero;
            raw[FMT == ROW_F32 ? 1 : 0] = valid && d0 + 4 < dim ? __ldg(src + 1) : zero;
        } else if (FMT == ROW_RABITQ) {
            // (64 sign bits per thread: see tile_scan_kernel)
        } else {
            const uint32_t per = FMT == ROW_SQ8 ? 16 : 8;
            const uint32_t d0 = piece * (8 * per) + kc * per;
            raw[0] = valid && d0 < dim ? __ldg(reinterpret_cast<const uint4*>(row + static_cast<size_t>(d0) * (FMT == ROW_SQ8 ? 1 : 2))) : zero;
        }
    }
    __device__ __forceinline__ void
    store(unsigned char* dst, uint32_t piece, uint32_t kc, uint32_t dim) const {
        if (FMT == ROW_F32) {
            float x[8];
            const uint4 a = raw[0], b = raw[FMT == ROW_F32 ? 1 : 0];
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
            const uint32_t d0 = piece * 64 + kc * 8;
#pragma unroll
            for (uint32_t i = 0; i < 8; ++i) {
                x[i] = d0 + i < dim ? __uint_as_float(w[i]) : 0.f;
            }
            uint4 hi, lo;
            split_bf16x8(x, hi, lo);
            *reinterpret_cast<uint4*>(dst) = hi;
            *reinterpret_cast<uint4*>(dst + TILE_A_TERM) = lo;
        } else if (FMT == ROW_SQ8) {
            *reinterpret_cast<uint4*>(dst) = make_uint4(raw[0].x ^ 0x80808080u, raw[0].y ^ 0x80808080u, raw[0].z ^ 0x80808080u,
                                                        raw[0].w ^ 0x80808080u);
        } else {
            uint32_t w[4] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w};
            const uint32_t d0 = piece * 64 + kc * 8;
            if (d0 + 8 > dim) {   // bytes past the last dimension are not defined
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    const uint32_t keep = (d0 + 2 * i < dim ? 0x0000FFFFu : 0u) | (d0 + 2 * i + 1 < dim ? 0xFFFF0000u : 0u);
                    w[i] &= keep;
                }
            }
            *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
};

// 8 consecutive 32-bit columns of this thread's TMEM lane.
__device__ __forceinline__ void
tmem_load_8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
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

// QT queries per item at most (16, 32 or 64).
template <int FMT, int QT>
__global__ void __launch_bounds__(TILE_THREADS, 1)
tile_scan_kernel(const TileScan p) {
    using F = TileFmt<FMT>;
    constexpr uint32_t N = F::B_TERMS * QT;                  // rows of B, columns of the accumulator
    constexpr uint32_t STAGE = F::A_TERMS * TILE_A_TERM;
    constexpr uint32_t B_PIECE = N * TILE_PIECE;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ TileShared sh;
    // the swizzle permutes by address bits: blocks start on 1 KiB
    unsigned char* const smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t stages = p.stages, pieces = p.pieces, dim = p.s.dim;
    unsigned char* const b_smem = smem + stages * STAGE;
    const uint32_t b_bytes = pieces * B_PIECE;
    const volatile uint32_t* failed = &sh.failed;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < stages; ++s) {
            mbar_init(&sh.full[s], TILE_LOAD_WARPS);
            mbar_init(&sh.freed[s], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&sh.b_full[i], TILE_LOAD_WARPS);
            mbar_init(&sh.b_free[i], 1);
            mbar_init(&sh.acc_full[i], 1);
            mbar_init(&sh.acc_free[i], TILE_EPI_WARPS);
        }
        sh.failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TILE_EPI_WARPS) {
        tmem_alloc(&sh.tmem_base, 2 * TILE_ACC_COLS);
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = sh.tmem_base;
    const uint32_t n_items = *p.n_items;
    bool ok = true;

    if (warp > TILE_EPI_WARPS) {
        // ---------------- loaders: code records -> operands ----------------
        const uint32_t lt = threadIdx.x - 32 * (TILE_EPI_WARPS + 1);
        const uint32_t lwarp = lt >> 5;
        constexpr uint32_t SETS = FMT == ROW_F32 ? 2 : 4;    // pieces requested ahead, in registers
        constexpr uint32_t UNITS = 1024 / TILE_LOADERS;      // 16-byte operand units per thread and piece
        // Where the loads are; items are dealt round-robin, and a cursor reads the next item's description while it
        // works through the current one.
        struct Cursor {
            uint32_t item, lbeg, len, pair0, nqt, next_lbeg, next_len, next_pair0, next_nqt, r0, piece;
        };
        auto describe = [&](uint32_t item, uint32_t& lbeg, uint32_t& len, uint32_t& pair0, uint32_t& nqt) {
            lbeg = len = pair0 = nqt = 0;
            if (item < n_items) {
                const uint4 d = __ldg(reinterpret_cast<const uint4*>(p.items + item));
                lbeg = __ldg(p.s.list_off + d.x) + d.w;
                len = min(__ldg(p.s.list_off + d.x + 1) - lbeg, TILE_SEGMENT);
                pair0 = d.y;
                nqt = d.z;
            }
        };
        auto start = [&](Cursor& c) {
            c.item = blockIdx.x;
            c.r0 = c.piece = 0;
            describe(c.item, c.lbeg, c.len, c.pair0, c.nqt);
            describe(c.item + gridDim.x, c.next_lbeg, c.next_len, c.next_pair0, c.next_nqt);
        };
        auto advance = [&](Cursor& c) {
            if (++c.piece < pieces) {
                return;
            }
            c.piece = 0;
            c.r0 += 128;
            if (c.r0 < c.len) {
                return;
            }
            c.r0 = 0;
            c.item += gridDim.x;
            c.lbeg = c.next_lbeg;
            c.len = c.next_len;
            c.pair0 = c.next_pair0;
            c.nqt = c.next_nqt;
            describe(c.item + gridDim.x, c.next_lbeg, c.next_len, c.next_pair0, c.next_nqt);
        };
        // eight lanes on the line of a row, four rows per warp and step
        const uint32_t kc = lane & 7u, rr = lwarp * (128 / TILE_LOAD_WARPS) + (lane >> 3);
        TileUnit<FMT> u[SETS][UNITS];
        auto request = [&](const Cursor& c, TileUnit<FMT> (&set)[UNITS]) {
            if (c.item >= n_items) {
                return;
            }
            const uint8_t* rows = p.s.codes + static_cast<uint64_t>(c.lbeg) * p.s.code_stride;
            if (FMT == ROW_RABITQ) {
                // a thread takes 64 dimensions of one row: eight bytes of sign bits, four k-cores
                const uint32_t r = c.r0 + (lt >> 1), part = lt & 1u;
                set[0].bits = r < c.len && c.piece * 128 + part * 64 < dim
                                  ? __ldg(reinterpret_cast<const uint2*>(rows + static_cast<uint64_t>(r) * p.s.code_stride + c.piece * 16 + part * 8))
                                  : make_uint2(0u, 0u);
                return;
            }
#pragma unroll
            for (uint32_t j = 0; j < UNITS; ++j) {
                const uint32_t r = c.r0 + rr + j * 4;
                set[j].load(rows + static_cast<uint64_t>(r < c.len ? r : 0u) * p.s.code_stride, r < c.len, c.piece, kc, dim);
            }
        };
        uint32_t stage = 0, phase = 0, filled = 0, n_mine = 0;
        auto load_queries = [&](const Cursor& c) -> bool {
            const uint32_t buf = p.b_bufs == 2 ? n_mine & 1u : 0u;
            if (n_mine >= p.b_bufs) {
                // (use number n_mine / b_bufs of this buffer: the use before it must have been multiplied)
                if (!tile_wait(&sh.b_free[buf], ((n_mine / p.b_bufs) - 1u) & 1u, failed, p.spin_limit, lane)) {
                    return false;
                }
            }
            unsigned char* bd = b_smem + buf * b_bytes;
            const uint32_t per_row = pieces * 8;             // units of a row of B
            if (F::INT8) {
#pragma unroll 4
                for (uint32_t i = lt; i < N * per_row; i += TILE_LOADERS) {
                    const uint32_t r = i / per_row, k = i - r * per_row;
                    const uint32_t term = r / QT, qi = r - term * QT;
                    uint4 v = make_uint4(0u, 0u, 0u, 0u);
                    if (qi < c.nqt && k * 16 < p.qstride) {
                        const uint32_t q = __ldg(p.pair_ids + c.pair0 + qi) / p.nprobe;
                        v = __ldg(reinterpret_cast<const uint4*>(p.qw8 + (static_cast<uint64_t>(q) * 3 + term) * p.qstride + k * 16));
                    }
                    *reinterpret_cast<uint4*>(bd + (k >> 3) * B_PIECE + swizzled(r, k & 7u)) = v;
                }
            } else {
#pragma unroll 2
                for (uint32_t i = lt; i < QT * per_row; i += TILE_LOADERS) {
                    const uint32_t qi = i / per_row, k = i - qi * per_row;
                    float x[8];
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        x[e] = 0.f;
                    }
                    if (qi < c.nqt) {
                        const uint32_t q = __ldg(p.pair_ids + c.pair0 + qi) / p.nprobe;
                        const float* src = p.s.queries + static_cast<uint64_t>(q) * dim + k * 8;
#pragma unroll
                        for (uint32_t e = 0; e < 8; ++e) {
                            x[e] = k * 8 + e < dim ? __ldg(src + e) : 0.f;
                        }
                    }
                    unsigned char* dst = bd + (k >> 3) * B_PIECE + swizzled(qi, k & 7u);
                    if (FMT == ROW_F32) {
                        uint4 hi, lo;
                        split_bf16x8(x, hi, lo);
                        *reinterpret_cast<uint4*>(dst) = hi;
                        *reinterpret_cast<uint4*>(dst + QT * 128) = lo;
                    } else {
                        constexpr int HF = FMT == ROW_BF16 ? SCAN_FMT_BF16 : SCAN_FMT_FP16;
                        uint32_t w[4];
#pragma unroll
                        for (uint32_t e = 0; e < 4; ++e) {
                            const uint32_t lo = qi < c.nqt && k * 8 + 2 * e < dim ? half_encode<HF>(x[2 * e]) : 0u;
                            const uint32_t hi = qi < c.nqt && k * 8 + 2 * e + 1 < dim ? half_encode<HF>(x[2 * e + 1]) : 0u;
                            w[e] = lo | (hi << 16);
                        }
                        *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
            tile_publish(&sh.b_full[buf], lane);
            ++n_mine;
            return true;
        };
        Cursor now, ahead;
        start(now);
        start(ahead);
#pragma unroll
        for (uint32_t s = 0; s < SETS; ++s) {
            request(ahead, u[s]);
            if (ahead.item < n_items) {
                advance(ahead);
            }
        }
        while (now.item < n_items && ok) {
#pragma unroll
            for (uint32_t s = 0; s < SETS; ++s) {
                if (now.item >= n_items || !ok) {
                    break;
                }
                if (now.r0 == 0 && now.piece == 0) {
                    ok = load_queries(now);
                }
                if (ok && filled >= stages) {
                    ok = tile_wait(&sh.freed[stage], phase ^ 1u, failed, p.spin_limit, lane);
                }
                if (!ok) {
                    break;
                }
                unsigned char* dst = smem + stage * STAGE;
                if (FMT == ROW_RABITQ) {
                    const uint32_t r = lt >> 1, part = lt & 1u;
                    const uint2 bits = u[s][0].bits;
                    *reinterpret_cast<uint4*>(dst + swizzled(r, part * 4)) = spread_bits16(bits.x & 0xFFFFu);
                    *reinterpret_cast<uint4*>(dst + swizzled(r, part * 4 + 1)) = spread_bits16(bits.x >> 16);
                    *reinterpret_cast<uint4*>(dst + swizzled(r, part * 4 + 2)) = spread_bits16(bits.y & 0xFFFFu);
                    *reinterpret_cast<uint4*>(dst + swizzled(r, part * 4 + 3)) = spread_bits16(bits.y >> 16);
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < UNITS; ++j) {
                        u[s][j].store(dst + swizzled(rr + j * 4, kc), now.piece, kc, dim);
                    }
                }
                tile_publish(&sh.full[stage], lane);
                request(ahead, u[s]);
                if (ahead.item < n_items) {
                    advance(ahead);
                }
                advance(now);
                ++filled;
                if (++stage == stages) {
                    stage = 0;
                    phase ^= 1u;
                }
            }
        }
    } else if (warp == TILE_EPI_WARPS) {
        // ---------------- MMA issue (one thread) ----------------
        if (lane == 0) {
            constexpr uint32_t idesc = F::INT8 ? umma_idesc_s8(128, N)
                                               : (FMT == ROW_FP16 ? umma_idesc_f16(128, N) : umma_idesc_bf16(128, N));
            constexpr uint32_t idesc_lo = umma_idesc_bf16(128, QT);   // fp32: lo terms of the rows against hi terms of the queries
            const uint64_t a0 = umma_desc_sw128(smem_u32(smem)), b0 = umma_desc_sw128(smem_u32(b_smem));
            uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0, tiles = 0, n_mine = 0;
            for (uint32_t item = blockIdx.x; item < n_items && ok; item += gridDim.x, ++n_mine) {
                const uint4 d = __ldg(reinterpret_cast<const uint4*>(p.items + item));
                const uint32_t len = min(__ldg(p.s.list_off + d.x + 1) - __ldg(p.s.list_off + d.x) - d.w, TILE_SEGMENT);
                const uint32_t buf = p.b_bufs == 2 ? n_mine & 1u : 0u;
                ok = tcs_wait(&sh.b_full[buf], (n_mine / p.b_bufs) & 1u, failed, p.spin_limit);
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
#pragma unroll
                        for (uint32_t ks = 0; ks < 4; ++ks) {
                            const uint32_t accumulate = (piece | ks) != 0 ? 1u : 0u;
                            if (F::INT8) {
                                umma_s8(d_tmem, a + ks * 2, b + ks * 2, idesc, accumulate);
                            } else {
                                umma_bf16(d_tmem, a + ks * 2, b + ks * 2, idesc, accumulate);
                            }
                            if (FMT == ROW_F32) {
                                umma_bf16(d_tmem, a + (TILE_A_TERM >> 4) + ks * 2, b + ks * 2, idesc_lo, 1u);
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
    } else {
        // ---------------- epilogue: one thread per row of the tile, two warps per 32 rows share the queries ----------------
        const uint32_t quarter = warp & 3u, half = warp >> 2;
        const uint32_t row = quarter * 32 + lane;
        uint32_t tile = 0;
        const bool filtered = p.s.filter_pos_inner != nullptr;
        for (uint32_t item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
            const uint4 d = __ldg(reinterpret_cast<const uint4*>(p.items + item));
            const uint32_t lbeg = __ldg(p.s.list_off + d.x) + d.w, len = min(__ldg(p.s.list_off + d.x + 1) - lbeg, TILE_SEGMENT);
            __syncwarp();
            for (uint32_t j = lane; j < QT; j += 32) {
                const bool used = j < d.z;
                const uint32_t pair = used ? __ldg(p.pair_ids + d.y + j) : 0u, q = pair / p.nprobe;
                sh.out[warp][j] = used ? q * p.t.stride + __ldg(p.t.base + pair) + d.w : 0u;
                if (FMT == ROW_SQ8) {
                    sh.c0[warp][j] = used ? __ldg(p.s.qa + q) : 0.f;
                    sh.c1[warp][j] = used ? p.s.coef_c * __ldg(p.qscale + q) : 0.f;
                } else if (FMT == ROW_RABITQ) {
                    sh.c0[warp][j] = used ? __ldg(p.s.queries + static_cast<uint64_t>(q) * (dim + 1) + dim) : 0.f;
                    sh.c1[warp][j] = used ? __ldg(p.qscale + q) : 0.f;
                    sh.t1[warp][j] = used ? __ldg(p.qsum + 4 * q) : 0;
                    sh.t2[warp][j] = used ? __ldg(p.qsum + 4 * q + 1) : 0;
                    sh.t3[warp][j] = used ? __ldg(p.qsum + 4 * q + 2) : 0;
                }
            }
            __syncwarp();
            for (uint32_t r0 = 0; r0 < len; r0 += 128, ++tile) {
                const uint32_t r = r0 + row, acc = tile & 1u;
                const bool valid = r < len;
                const uint32_t pos = lbeg + (valid ? r : 0u);
                // what the row contributes to its scores
                float x0 = 0.f, x1 = 1.f;
                if (FMT == ROW_SQ8) {
                    x0 = p.s.coef_b * __ldg(p.s.code_norm + pos);
                } else if (FMT == ROW_RABITQ) {
                    const float* tail = reinterpret_cast<const float*>(p.s.codes + static_cast<uint64_t>(pos) * p.s.code_stride + p.s.dpad / 8);
                    x0 = __ldg(tail);
                    x1 = __ldg(tail + 1);
                    if (fabsf(x1) < 1e-5f) {
                        x1 = x1 >= 0.f ? 1.0f : -1.0f;
                    }
                    x1 = -2.0f * x0 / x1;
                    x0 *= x0;
                } else if (p.l2 != 0) {
                    x0 = __ldg(p.row_norm + pos);
                }
                const bool drop = !valid || (filtered && scan_row_filtered(p.s, pos));
                ok = tile_wait(&sh.acc_full[acc], (tile >> 1) & 1u, failed, p.spin_limit, lane);
                if (!ok) {
                    break;
                }
                tc_fence_after_sync();
                const uint32_t taddr = tmem_base + ((quarter * 32u) << 16) + acc * TILE_ACC_COLS;
                if (r0 + quarter * 32 < len) {   // (the warp's rows are one group of 32 scores)
                    // the last read of an accumulator is followed by its hand-over; columns past the item's queries hold
                    // products with zero and are not stored
                    for (uint32_t g = half * 8; g < d.z; g += 16) {
                        uint32_t v1[8], v2[8], v3[8];
                        tmem_load_8(taddr + g, v1);
                        if (F::B_TERMS >= 2) {
                            tmem_load_8(taddr + QT + g, v2);
                        }
                        if (F::B_TERMS >= 3) {
                            tmem_load_8(taddr + 2 * QT + g, v3);
                        }
                        tmem_load_wait();
                        float v[8];
#pragma unroll
                        for (uint32_t i = 0; i < 8; ++i) {
                            const uint32_t j = g + i;
                            if (FMT == ROW_SQ8) {
                                const float low = static_cast<float>(static_cast<int32_t>(v2[i]) * 254 + static_cast<int32_t>(v3[i]));
                                const float f = fmaf(low, 1.0f / 64516.0f, static_cast<float>(static_cast<int32_t>(v1[i])));
                                v[i] = fmaf(sh.c1[warp][j], f, x0) + sh.c0[warp][j];
                            } else if (FMT == ROW_RABITQ) {
                                // |x|^2 + |q|^2 - 2 |x| |q| (ip / error); the set bits' sum S gives ip = 2 S - (sum of all)
                                const int32_t u1 = 2 * static_cast<int32_t>(v1[i]) - sh.t1[warp][j];
                                const int32_t u2 = 2 * static_cast<int32_t>(v2[i]) - sh.t2[warp][j];
                                const int32_t u3 = 2 * static_cast<int32_t>(v3[i]) - sh.t3[warp][j];
                                const float f = fmaf(static_cast<float>(u2 * 254 + u3), 1.0f / 64516.0f, static_cast<float>(u1));
                                const float qn = sh.c0[warp][j];
                                v[i] = fmaf(x1 * qn, f * sh.c1[warp][j], fmaf(qn, qn, x0));
                            } else {
                                float ip = __uint_as_float(v1[i]);
                                if (FMT == ROW_F32) {
                                    ip += __uint_as_float(v2[i]);
                                }
                                v[i] = p.l2 != 0 ? fmaf(-2.0f, ip, x0) : -ip;
                            }
                        }
                        uint32_t least = 0;   // of column g + lane
#pragma unroll
                        for (uint32_t i = 0; i < 8; ++i) {
                            const uint32_t bits = drop ? SCORE_FILTERED : __float_as_uint(v[i]);
                            if (g + i < d.z) {
                                reinterpret_cast<uint32_t*>(p.t.scores)[sh.out[warp][g + i] + r] = bits;
                            }
                            const uint32_t low = __reduce_min_sync(0xffffffffu, ScoreSource<>::ordered(bits));
                            least = lane == i ? low : least;
                        }
                        if (lane < 8 && g + lane < d.z) {
                            p.t.minima[(sh.out[warp][g + lane] + r0 + quarter * 32) >> 5] = least;
                        }
                    }
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sh.acc_free[acc]);
                }
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
        tc_drain_pause();   // a wait gave up: let the MMAs still in flight land before the CTA lets go
        __syncthreads();
    }
    if (warp == TILE_EPI_WARPS) {
        tmem_dealloc(tmem_base, 2 * TILE_ACC_COLS);
    }
}

}  // namespace vb200
