// Scans of contiguous rows by a thread per row: the building block of every search that meets too little reuse
// for tensor-core tiles -- a few queries against the probed lists, the routing distances of a small batch, exact
// search for a handful of queries.
//
// Each thread owns one row and walks its dimensions upward, so the fp32 and half-precision codecs and the one-bit
// estimator come out as the reference's own operation chains: the values are final and no re-scoring follows
// (SQ8 ranks with the exact integer sums of the int8 weight terms and is re-scored).  A thread that fetched its
// own row would touch one sector of 32 different lines per load; instead a CTA moves pieces of RS_PIECE bytes of
// its 128 rows through shared memory with asynchronous copies, neighbouring lanes on neighbouring 16 bytes, three
// pieces deep.  Rows in shared memory are 16 bytes apart modulo 128, so the 16-byte reads are free of conflicts.
#pragma once

#include "dense.cuh"
#include "ivf_scan.cuh"
#include "tc_gemm.cuh"

namespace vb200 {

constexpr int RS_ROWS = 128;                       // rows per chunk = threads per CTA
constexpr uint32_t RS_PIECE = 128;                 // bytes of a row per stage
constexpr uint32_t RS_STRIDE = RS_PIECE + 16;
constexpr uint32_t RS_STAGE = RS_ROWS * RS_STRIDE;
constexpr int RS_STAGES = 3;

enum RowFmt { ROW_F32 = 0, ROW_BF16 = 1, ROW_FP16 = 2, ROW_SQ8 = 3, ROW_RABITQ = 4,
              ROW_F32_SPLIT = 5 };   // (tiles only: fp32 rows as two bf16 terms)

// What a thread accumulates over its row for QN queries.  `unit` consumes 16 bytes of the row that start at
// dimension d0; `tail` the same when fewer than a whole unit of dimensions is left.
template <int FMT, bool L2, int QN>
struct RowAcc {   // fp32 / bf16 / fp16 rows: the chain over ascending dimensions
    static constexpr uint32_t UNIT_DIMS = FMT == ROW_F32 ? 4 : 8;
    float acc[QN];
    __device__ __forceinline__ void
    clear() {
#pragma unroll
        for (int i = 0; i < QN; ++i) {
            acc[i] = 0.f;
        }
    }
    __device__ __forceinline__ static void
    decode(const uint4& w, float* x) {
        const uint32_t v[4] = {w.x, w.y, w.z, w.w};
        if (FMT == ROW_F32) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                x[i] = __uint_as_float(v[i]);
            }
        } else {
            constexpr int F = FMT == ROW_BF16 ? SCAN_FMT_BF16 : SCAN_FMT_FP16;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                x[(2 * i) & (static_cast<int>(UNIT_DIMS) - 1)] = half_decode<F>(v[i] & 0xFFFFu);
                x[(2 * i + 1) & (static_cast<int>(UNIT_DIMS) - 1)] = half_decode<F>(v[i] >> 16);
            }
        }
    }
    __device__ __forceinline__ static void
    step(float& a, float x, float q) {
        if (L2) {
            const float t = __fsub_rn(x, q);
            a = fmaf(t, t, a);
        } else {
            a = fmaf(x, q, a);
        }
    }
    __device__ __forceinline__ void
    unit(const uint4& w, const float* q, uint32_t qstride, uint32_t d0) {
        float x[UNIT_DIMS];
        decode(w, x);
#pragma unroll
        for (int i = 0; i < QN; ++i) {
#pragma unroll
            for (uint32_t j = 0; j < UNIT_DIMS; j += 4) {
                const float4 v = *reinterpret_cast<const float4*>(q + i * qstride + d0 + j);
                step(acc[i], x[j], v.x);
                step(acc[i], x[j + 1], v.y);
                step(acc[i], x[j + 2], v.z);
                step(acc[i], x[j + 3], v.w);
            }
        }
    }
    __device__ __forceinline__ void
    tail(const uint4& w, const float* q, uint32_t qstride, uint32_t d0, uint32_t left) {
        float x[UNIT_DIMS];
        decode(w, x);
#pragma unroll
        for (uint32_t j = 0; j < UNIT_DIMS; ++j) {
            if (j < left) {
#pragma unroll
                for (int i = 0; i < QN; ++i) {
                    step(acc[i], x[j], q[i * qstride + d0 + j]);
                }
            }
        }
    }
};

// SQ8: the sum over the three int8 terms of a query's weights, a1 + a2 / 254 + a3 / 254^2, from the exact integer sums.
// 254 a2 + a3 reaches 127 * 128 * 255 per dimension, so it fits 32 bits up to 518 dimensions; longer rows add the two as
// floats, whose rounding (2^-24 of a2 / 254) is far below what the terms themselves leave out.
constexpr uint32_t SQ8_NARROW_DIMS = 518;

__device__ __forceinline__ float
sq8_term_sum(int32_t a1, int32_t a2, int32_t a3, bool narrow) {
    const float low = narrow ? static_cast<float>(a2 * 254 + a3) : fmaf(static_cast<float>(a2), 254.0f, static_cast<float>(a3));
    return fmaf(low, 1.0f / 64516.0f, static_cast<float>(a1));
}

// Three integer sums over the int8 weight terms of each of QN queries, [QN][3][qstride] bytes behind `q`; terms past the
// last dimension are zero.  `live`: queries there are (the others cost a test).
template <bool L2, int QN>
struct RowAcc<ROW_SQ8, L2, QN> {
    static constexpr uint32_t UNIT_DIMS = 16;
    int32_t a1[QN], a2[QN], a3[QN];
    uint32_t live = QN;
    __device__ __forceinline__ void
    clear() {
#pragma unroll
        for (int i = 0; i < QN; ++i) {
            a1[i] = a2[i] = a3[i] = 0;
        }
    }
    __device__ __forceinline__ void
    unit(const uint4& w, const float* q, uint32_t qstride, uint32_t d0) {
        const int c0 = static_cast<int>(w.x ^ 0x80808080u), c1 = static_cast<int>(w.y ^ 0x80808080u),
                  c2 = static_cast<int>(w.z ^ 0x80808080u), c3 = static_cast<int>(w.w ^ 0x80808080u);
#pragma unroll
        for (int i = 0; i < QN; ++i) {
            if (QN > 1 && static_cast<uint32_t>(i) >= live) {
                break;
            }
            const int8_t* t = reinterpret_cast<const int8_t*>(q) + i * 3 * qstride + d0;
            const int4 t1 = *reinterpret_cast<const int4*>(t), t2 = *reinterpret_cast<const int4*>(t + qstride),
                       t3 = *reinterpret_cast<const int4*>(t + 2 * qstride);
            a1[i] = __dp4a(c0, t1.x, a1[i]);
            a2[i] = __dp4a(c0, t2.x, a2[i]);
            a3[i] = __dp4a(c0, t3.x, a3[i]);
            a1[i] = __dp4a(c1, t1.y, a1[i]);
            a2[i] = __dp4a(c1, t2.y, a2[i]);
            a3[i] = __dp4a(c1, t3.y, a3[i]);
            a1[i] = __dp4a(c2, t1.z, a1[i]);
            a2[i] = __dp4a(c2, t2.z, a2[i]);
            a3[i] = __dp4a(c2, t3.z, a3[i]);
            a1[i] = __dp4a(c3, t1.w, a1[i]);
            a2[i] = __dp4a(c3, t2.w, a2[i]);
            a3[i] = __dp4a(c3, t3.w, a3[i]);
        }
    }
    __device__ __forceinline__ void
    tail(const uint4& w, const float* q, uint32_t qstride, uint32_t d0, uint32_t) {
        unit(w, q, qstride, d0);
    }
};

// One-bit codes: the reference's chain of +-sv_d additions (ivf_rabitq_scan_kernel); sv is zero past the last
// dimension.  The two trailing floats of a record are read by the caller.
template <bool L2, int QN>
struct RowAcc<ROW_RABITQ, L2, QN> {
    static constexpr uint32_t UNIT_DIMS = 128;
    float acc[1];
    __device__ __forceinline__ void
    clear() {
        acc[0] = 0.f;
    }
    __device__ __forceinline__ void
    word(uint32_t w, const float* q) {
#pragma unroll
        for (int b4 = 0; b4 < 8; ++b4) {
            const uint32_t n = ~w >> (4 * b4);
            const float4 v = *reinterpret_cast<const float4*>(q + 4 * b4);
            acc[0] = fmaf(v.x, __uint_as_float(0x3F800000u | ((n & 1u) << 31)), acc[0]);
            acc[0] = fmaf(v.y, __uint_as_float(0x3F800000u | ((n & 2u) << 30)), acc[0]);
            acc[0] = fmaf(v.z, __uint_as_float(0x3F800000u | ((n & 4u) << 29)), acc[0]);
            acc[0] = fmaf(v.w, __uint_as_float(0x3F800000u | ((n & 8u) << 28)), acc[0]);
        }
    }
    __device__ __forceinline__ void
    unit(const uint4& w, const float* q, uint32_t, uint32_t d0) {
        word(w.x, q + d0);
        word(w.y, q + d0 + 32);
        word(w.z, q + d0 + 64);
        word(w.w, q + d0 + 96);
    }
    __device__ __forceinline__ void
    tail(const uint4& w, const float* q, uint32_t, uint32_t d0, uint32_t left) {
        word(w.x, q + d0);
        if (left > 32) {
            word(w.y, q + d0 + 32);
        }
        if (left > 64) {
            word(w.z, q + d0 + 64);
        }
        if (left > 96) {
            word(w.w, q + d0 + 96);
        }
    }
};

template <uint32_t N>
__device__ __forceinline__ void
cp_async_wait_group() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Copies bytes [k0, k0 + kb) of `rows` rows into a stage.  UNIT: bytes per copy the rows' alignment allows (16, 4,
// or 2 -- then through registers).  kb need not be a multiple of UNIT when UNIT is 16: the row is then readable up
// to the next multiple (index records are padded to 16 bytes).
template <int UNIT>
__device__ __forceinline__ void
row_stage_copy(unsigned char* stage, const unsigned char* src, uint64_t row_stride, uint32_t rows, uint32_t k0, uint32_t kb) {
    const uint32_t units = (kb + UNIT - 1) / UNIT;
    constexpr uint32_t FULL = RS_PIECE / UNIT;
    const uint32_t total = rows * units;
    for (uint32_t u = threadIdx.x; u < total; u += RS_ROWS) {
        const uint32_t r = units == FULL ? u / FULL : u / units;
        const uint32_t c = u - r * units;
        const unsigned char* from = src + r * row_stride + k0 + c * UNIT;
        unsigned char* to = stage + r * RS_STRIDE + c * UNIT;
        if (UNIT == 16) {
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(to)), "l"(from) : "memory");
        } else if (UNIT == 4) {
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(to)), "l"(from) : "memory");
        } else {
            *reinterpret_cast<uint16_t*>(to) = *reinterpret_cast<const uint16_t*>(from);
        }
    }
}

// Walks chunks first, first + step, ... of RS_ROWS rows each: per chunk every thread accumulates its row into acc
// and `emit(row, valid)` is called by all threads (it may contain barriers).
template <int UNIT, typename Acc, typename Emit>
__device__ __forceinline__ void
row_stream(const unsigned char* base, uint64_t row_stride, uint32_t row_bytes, uint32_t dim, uint64_t n_rows, uint64_t first,
           uint64_t step, unsigned char* stages, const float* q, uint32_t qstride, Acc& acc, Emit emit) {
    const uint64_t n_chunks = (n_rows + RS_ROWS - 1) / RS_ROWS;
    if (first >= n_chunks) {
        return;
    }
    const uint32_t mine = static_cast<uint32_t>((n_chunks - first + step - 1) / step);
    const uint32_t per_row = (row_bytes + RS_PIECE - 1) / RS_PIECE;
    const uint32_t total = mine * per_row;
    uint32_t i_chunk = 0, i_piece = 0;   // the next piece to request
    auto request = [&](uint32_t p) {
        if (p < total) {
            const uint64_t row0 = (first + static_cast<uint64_t>(i_chunk) * step) * RS_ROWS;
            const uint32_t rows = n_rows - row0 < RS_ROWS ? static_cast<uint32_t>(n_rows - row0) : RS_ROWS;
            const uint32_t k0 = i_piece * RS_PIECE;
            const uint32_t kb = row_bytes - k0 < RS_PIECE ? row_bytes - k0 : RS_PIECE;
            row_stage_copy<UNIT>(stages + (p % RS_STAGES) * RS_STAGE, base + row0 * row_stride, row_stride, rows, k0, kb);
            if (++i_piece == per_row) {
                i_piece = 0;
                ++i_chunk;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < RS_STAGES - 1; ++s) {
        request(s);
    }
    uint32_t piece = 0, chunk = 0;
    acc.clear();
    for (uint32_t p = 0; p < total; ++p) {
        cp_async_wait_group<RS_STAGES - 2>();
        __syncthreads();   // piece p is here for everybody, and nobody reads piece p - 1 any more
        request(p + RS_STAGES - 1);
        const unsigned char* mine_row = stages + (p % RS_STAGES) * RS_STAGE + threadIdx.x * RS_STRIDE;
        const uint32_t d_piece = piece * (RS_PIECE / 16) * Acc::UNIT_DIMS;
        const uint32_t d_left = dim - d_piece;
        if (d_left >= (RS_PIECE / 16) * Acc::UNIT_DIMS) {
#pragma unroll
            for (uint32_t j = 0; j < RS_PIECE / 16; ++j) {
                acc.unit(*reinterpret_cast<const uint4*>(mine_row + j * 16), q, qstride, d_piece + j * Acc::UNIT_DIMS);
            }
        } else {
            uint32_t j = 0;
            for (; (j + 1) * Acc::UNIT_DIMS <= d_left; ++j) {
                acc.unit(*reinterpret_cast<const uint4*>(mine_row + j * 16), q, qstride, d_piece + j * Acc::UNIT_DIMS);
            }
            if (j * Acc::UNIT_DIMS < d_left) {
                acc.tail(*reinterpret_cast<const uint4*>(mine_row + j * 16), q, qstride, d_piece + j * Acc::UNIT_DIMS,
                         d_left - j * Acc::UNIT_DIMS);
            }
        }
        if (++piece == per_row) {
            piece = 0;
            const uint64_t row = (first + static_cast<uint64_t>(chunk) * step) * RS_ROWS + threadIdx.x;
            emit(row, row < n_rows);
            ++chunk;
            acc.clear();
        }
    }
    cp_async_wait_group<0>();
}

// ---- distances of scattered rows by one warp ------------------------------------------------------------------
// A lane that walks a row of its own asks with every load for one sector each of 32 lines, and what bounds such a kernel is the L1
// cache taking them one by one (72 rows of 384 bytes per query, 10,000 queries: 82 % of its rate, 155 us with the selection before
// it; 97 this way).  Here the warp copies pieces of 128 bytes of 32 rows into shared memory, neighbouring lanes on
// neighbouring 16 bytes, a piece ahead, and each lane walks its row there.
constexpr uint32_t WARP_ROWS_STAGE = 32 * RS_STRIDE;
constexpr uint32_t WARP_ROWS_BYTES = 2 * WARP_ROWS_STAGE;   // shared memory of a warp, 16-byte aligned

// For i = 0 .. count - 1 (lane i % 32): acc over row(i), a 16-byte aligned record readable to the next multiple of 16 behind row_bytes,
// then emit(i, acc).  q: as for row_stream.
template <typename Acc, typename Row, typename Emit>
__device__ __forceinline__ void
warp_rows(uint32_t count, const Row& row, uint32_t row_bytes, uint32_t dim, const float* q, uint32_t qstride, unsigned char* stages, uint32_t lane,
          Acc& acc, const Emit& emit) {
    const uint32_t pieces = (row_bytes + RS_PIECE - 1) / RS_PIECE, batches = (count + 31) / 32, total = pieces * batches;
    uint32_t a_batch = 0, a_piece = 0;   // asked for next
    auto request = [&](uint32_t step) {
        if (step < total) {
            unsigned char* to = stages + (step & 1u) * WARP_ROWS_STAGE;
            const uint32_t k0 = a_piece * RS_PIECE, units = (min(row_bytes - k0, RS_PIECE) + 15) / 16;
            const uint32_t rows = min(count - a_batch * 32, 32u);
            const uint32_t c = lane & 7u;
            for (uint32_t r = lane >> 3; r < rows; r += 4) {
                if (c < units) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(to + r * RS_STRIDE + c * 16)),
                                 "l"(row(a_batch * 32 + r) + k0 + c * 16)
                                 : "memory");
                }
            }
            if (++a_piece == pieces) {
                a_piece = 0;
                ++a_batch;
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    request(0);
    uint32_t piece = 0, batch = 0;
    acc.clear();
    for (uint32_t step = 0; step < total; ++step) {
        request(step + 1);
        cp_async_wait_group<1>();
        __syncwarp();   // the piece is here for all lanes
        const unsigned char* mine = stages + (step & 1u) * WARP_ROWS_STAGE + lane * RS_STRIDE;
        const uint32_t d0 = piece * (RS_PIECE / 16) * Acc::UNIT_DIMS, left = dim - d0;
        if (left >= (RS_PIECE / 16) * Acc::UNIT_DIMS) {
#pragma unroll
            for (uint32_t j = 0; j < RS_PIECE / 16; ++j) {
                acc.unit(*reinterpret_cast<const uint4*>(mine + j * 16), q, qstride, d0 + j * Acc::UNIT_DIMS);
            }
        } else {
            uint32_t j = 0;
            for (; (j + 1) * Acc::UNIT_DIMS <= left; ++j) {
                acc.unit(*reinterpret_cast<const uint4*>(mine + j * 16), q, qstride, d0 + j * Acc::UNIT_DIMS);
            }
            if (j * Acc::UNIT_DIMS < left) {
                acc.tail(*reinterpret_cast<const uint4*>(mine + j * 16), q, qstride, d0 + j * Acc::UNIT_DIMS, left - j * Acc::UNIT_DIMS);
            }
        }
        if (++piece == pieces) {
            piece = 0;
            if (batch * 32 + lane < count) {
                emit(batch * 32 + lane, acc);
            }
            ++batch;
            acc.clear();
        }
        __syncwarp();   // nobody reads the piece any more
    }
    cp_async_wait_group<0>();
    __syncwarp();
}

// Distance of one row to the query (widened, in shared memory), rows fetched sixteen bytes at a time with eight
// loads in flight where their alignment allows.
template <typename E>
__device__ __forceinline__ float
row_exact_distance(const E* __restrict__ x, const float* qf, uint32_t dim, bool l2) {
    constexpr uint32_t VEC = 16 / sizeof(E);
    float s = 0.f;
    auto step = [&](float v, float q) {
        if (l2) {
            const float t = __fsub_rn(v, q);
            s = fmaf(t, t, s);
        } else {
            s = fmaf(v, q, s);
        }
    };
    if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0 && dim % VEC == 0) {
        const uint4* xv = reinterpret_cast<const uint4*>(x);
        const uint32_t nv = dim / VEC;
        for (uint32_t v0 = 0; v0 < nv; v0 += 8) {
            uint4 w[8];
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) {
                w[u] = v0 + u < nv ? __ldg(xv + v0 + u) : make_uint4(0, 0, 0, 0);
            }
#pragma unroll
            for (uint32_t u = 0; u < 8; ++u) {
                if (v0 + u < nv) {
                    E e[VEC];
                    *reinterpret_cast<uint4*>(e) = w[u];
#pragma unroll
                    for (uint32_t j = 0; j < VEC; ++j) {
                        step(widen(e[j]), qf[(v0 + u) * VEC + j]);
                    }
                }
            }
        }
    } else {
        for (uint32_t d = 0; d < dim; ++d) {
            step(widen(x[d]), qf[d]);
        }
    }
    return l2 ? s : __fsub_rn(1.0f, s);
}

}  // namespace vb200
