// Batched binary64 Cholesky factorisation in 64-bit fixed point (fix64.cuh), 16 < n <= 512, sm_103a.
//
// Reference: blast::potrf (dense/Potrf.hpp:66-106): left-looking; a column strip takes the products
// of all earlier columns (the ger(-1, ...) loop), is factored on the diagonal and solved below it.
//
// What bounds it: in binary64 the multiply-adds, 2 lanes a clock and SM whatever the mapping (33.6 ms for
// 2,048 matrices with n uniform in 64 .. 512, factored and solved with one right-hand side). In fixed point,
// with the matrix's rows scaled, the products of earlier columns run on the integer pipe (n <= 128) or on the
// tensor cores (above), which took the same batch to 9.3 ms and, for its n > 128, to 7.6 ms; binary64 is left
// with one conversion per factor entry, and with what cannot be certified. At n = 512 with three CTAs an SM, three quarters of a CTA's time are
// the products (tensor pipe 63% busy meanwhile, the rest taking entries apart into digits and waiting for
// the staged columns), 8% the diagonal blocks, 8% the rows below them, 7% the conversion. At n = 128
// the products are half, the diagonal blocks' chains a quarter.
//
// Mapping: one CTA of T threads per matrix, panels of 16 columns, the rows of a panel in chunks of T.
//  * Products, T = 32 and 64: each thread holds a 4 x 4 tile of the T x 16 chunk (rows T/4 apart, adjacent
//    columns; 64 registers of sums), the earlier columns come through shared memory 16 at a time, double
//    buffered with cp.async. A step costs 48 multiply-adds against 4 row loads and 2 (16-byte) column
//    loads, all free of bank conflicts.
//  * Products, T = 128: digits of 8 bits on the tensor cores (update_chunk_mma), 32 columns at a time. With
//    T = 64 this lost to the integer products (n = 128 x 4,000: 2.06 against 1.72 ms): six CTAs an SM for
//    eight.
//  * The first chunk's first 32 rows: one warp, a row per lane, the 16 columns right-looking in
//    registers, the pivot row's limbs by shuffles. The reciprocal square root is integer as well.
//  * Other rows: a row per thread against the diagonal block, right-looking in registers.
//  * A row of a panel that cannot be certified (fix64.cuh) is not stored. After its chunk the columns so far
//    become binary64, and what is left of the matrix is factored in binary64 (potrf_strips.cuh).
//  * The factor stays in fixed point in the workspace (L itself, unless the caller says otherwise), as
//    limbs or as digits, where the later panels read it, and becomes binary64 in one last pass.
//
// Panels of 16 keep the work inside a panel, which runs at a lower rate, at 8 n^2 of the n^3 / 6
// products, and let all T threads own a row of it.
#include "common.cuh"
#include "fix64.cuh"
#include "potrf_strips.cuh"

namespace blastgpu {
namespace {

using fix64::Limbs;
using fix64::Rsqrt;

constexpr int kNB = 16;

template <int T>
struct Shape {
    static constexpr int NMAX = T == 32 ? 64 : T == 64 ? 128 : 512;  // largest n that runs with T threads
    static constexpr bool kTensor = T == 128;  // products on the tensor cores
    static constexpr int kWarps = T / 32;
    static constexpr int RT = T / 4;  // distance of a thread's rows in integer products
    // staged column: the chunk's rows, then the diagonal block's (reads of 8 rows by 2 columns hit all banks)
    static constexpr int RS = T + kNB + (kTensor ? 4 : 0);
    static constexpr int CS = T + 2;        // column stride of the chunk's remainders
    static constexpr int kStage = 0;
    static constexpr int kDigits = kStage + 2 * kNB * RS * 8;
    static constexpr int kChunk = kDigits + (kTensor ? 2 * 8 * kNB * kNB * 2 : 0);
    static constexpr int kDiag = kChunk + kNB * CS * 8;
    static constexpr int kRsqrt = kDiag + kNB * kNB * 8;
    static constexpr int kScale = kRsqrt + kNB * 16;
    static constexpr int kRow = kScale + NMAX * 2;
    static constexpr int kBytes = kRow + NMAX * 4;
    // solve_row reads past the diagonal block's last row: rows up to 18.
    static_assert(kDiag + 8 * (18 * kNB + kNB) <= kBytes);
};

template <int T>
__device__ __forceinline__ void cta_sync() {
    if constexpr (T == 32) __syncwarp();
    else __syncthreads();
}

__device__ __forceinline__ void cp_async8(int64_t* dst, const int64_t* src) {
    unsigned const d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

// Columns 16 s .. 16 s + 15 of the workspace, rows k0 + r0 .. of the chunk; below the first chunk
// also the diagonal block's rows.
template <int T>
__device__ __forceinline__ void stage_columns(int64_t* stage, const int64_t* W, int64_t ldw, int k0, int r0, int mr, int nb,
                                              int s) {
    using S = Shape<T>;
    int64_t* dst = stage + (s & 1) * kNB * S::RS;
    int64_t const* src = W + k0 + (int64_t)(kNB * s) * ldw;
    int const tid = threadIdx.x;
    if (tid < mr) {
#pragma unroll
        for (int q = 0; q < kNB; ++q) cp_async8(dst + q * S::RS + tid, src + r0 + tid + q * ldw);
    }
    if (r0 > 0) {
        for (int e = tid; e < kNB * kNB; e += T) {
            int const q = e / kNB, r = e % kNB;
            if (r < nb) cp_async8(dst + q * S::RS + T + r, src + r + q * ldw);
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// Digit i (0 the highest) of two entries as a pair of binary16 numbers: the byte becomes the low bits of
// 1024 + byte, and 1152 is taken off again.
template <int I>
__device__ __forceinline__ uint32_t digit_pair(int64_t u0, int64_t u1) {
    uint32_t const a = I < 4 ? (uint32_t)(u0 >> 32) : (uint32_t)u0, b = I < 4 ? (uint32_t)(u1 >> 32) : (uint32_t)u1;
    constexpr int kByte = 3 - (I & 3);
    uint32_t const bytes = __byte_perm(a, b, kByte | kByte << 4 | (4 + kByte) << 8 | (4 + kByte) << 12);
    uint32_t const biased = (bytes & 0x00ff00ffu) | 0x64006400u;
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(biased), "r"(0x64806480u));
    return d;
}
__device__ __forceinline__ void digit_pairs(uint32_t (&d)[8], int64_t u0, int64_t u1) {
    d[0] = digit_pair<0>(u0, u1), d[1] = digit_pair<1>(u0, u1), d[2] = digit_pair<2>(u0, u1), d[3] = digit_pair<3>(u0, u1);
    d[4] = digit_pair<4>(u0, u1), d[5] = digit_pair<5>(u0, u1), d[6] = digit_pair<6>(u0, u1), d[7] = digit_pair<7>(u0, u1);
}

__device__ __forceinline__ void mma_f16(float (&c)[4], uint32_t const (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// The chunk's remainders A - L L^T over the columns before k0, into C (units of 2^-62). RA: rows per
// thread that the chunk needs. Rows past mr and columns past nb hold whatever shared memory held; they
// are not used.
template <int T, int RA>
__device__ __forceinline__ void update_chunk_int(int k0, int r0, int mr, int nb, const double* A, int64_t lda,
                                             const int64_t* W, int64_t ldw, int64_t* stage, int64_t* C, const short* scale,
                                             uint32_t* row) {
    using S = Shape<T>;
    int const lane = threadIdx.x & 31, ct = 4 * (lane >> 3), rt = 8 * (threadIdx.x >> 5) + (lane & 7);
    int const slabs = k0 / kNB;
    if (slabs > 0) stage_columns<T>(stage, W, ldw, k0, r0, mr, nb, 0);
    double a[RA][4];
#pragma unroll
    for (int i = 0; i < RA; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int const r = rt + S::RT * i, c = ct + j;
            a[i][j] = (r < mr && c < nb && r0 + r >= c) ? A[(k0 + r0 + r) + (int64_t)(k0 + c) * lda] : 0.0;
        }
    int64_t hh[RA][4], cr[RA][4];
#pragma unroll
    for (int i = 0; i < RA; ++i) {
        int const r = rt + S::RT * i;
        int const er = r < mr ? scale[k0 + r0 + r] : 0;
        bool ok = true;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int const ec = ct + j < nb ? scale[k0 + ct + j] : 0;
            int64_t v;
            ok &= fix64::from_double(a[i][j], er + ec, v);
            hh[i][j] = -v;
            cr[i][j] = fix64::kCrossStart;
        }
        if (!ok && r < mr) atomicOr(row + k0 + r0 + r, fix64::kTodo);
    }
    int64_t const* colbase = stage + (r0 == 0 ? ct : T + ct);
    int64_t const* rowbase = stage + rt;
    for (int s = 0; s < slabs; ++s) {
        if (s + 1 < slabs) {
            stage_columns<T>(stage, W, ldw, k0, r0, mr, nb, s + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        cta_sync<T>();
        int const base = (s & 1) * kNB * S::RS;
#pragma unroll 4
        for (int q = 0; q < kNB; ++q) {
            int4 const b01 = *reinterpret_cast<int4 const*>(colbase + base + q * S::RS);
            int4 const b23 = *reinterpret_cast<int4 const*>(colbase + base + q * S::RS + 2);
            int const bl[4] = {b01.x, b01.z, b23.x, b23.z}, bh[4] = {b01.y, b01.w, b23.y, b23.w};
#pragma unroll
            for (int i = 0; i < RA; ++i) {
                Limbs const v = fix64::unpack(rowbase[base + q * S::RS + S::RT * i]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    fix64::mad(hh[i][j], v.h, bh[j]);
                    fix64::mad(cr[i][j], v.h, bl[j]);
                    fix64::mad(cr[i][j], v.l, bh[j]);
                }
            }
        }
        if ((s & 1) != 0) {  // fix64::kFold terms since the last time
#pragma unroll
            for (int i = 0; i < RA; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) fix64::fold(hh[i][j], cr[i][j]);
        }
        cta_sync<T>();  // this half is staged again two slabs on
    }
#pragma unroll
    for (int i = 0; i < RA; ++i) {
        int const r = rt + S::RT * i;
        if (r < mr) {
#pragma unroll
            for (int j = 0; j < 4; ++j) C[(ct + j) * S::CS + r] = -fix64::total(hh[i][j], cr[i][j]);
        }
    }
}

// The same on the tensor cores. An entry is 8 digits of 8 bits; the 36 products of digits i + j <= 7 go into 8
// binary32 accumulators by i + j. All are sums of integers: over 32 columns, 6 products of at most 2^14 and 2
// of at most 2^13 (an entry's highest digit has 6 bits) a column stay below 2^22, so they are exact, and an
// accumulator that starts at 1.5 x 2^23 holds its sum in its low mantissa bits. The digits i + j > 7 left out
// weigh 2^-60 sqrt(columns) in all.
// Warp w has the row tiles (16 rows) w and w + T/32; lane (g, q) = (lane / 4, lane % 4) of a tile has rows g, g + 8
// and columns 2 q, 2 q + 1 of each 8 columns. The 16 rows of the diagonal block are taken apart into digits
// once per 32 columns, by all threads, in fragment order; a row tile's by the warp that has it.
template <int T>
__device__ __forceinline__ void update_chunk_mma(int k0, int r0, int mr, int nb, const double* A, int64_t lda,
                                                 const int64_t* W, int64_t ldw, int64_t* stage, uint4* digits, int64_t* C,
                                                 const short* scale, uint32_t* row) {
    using S = Shape<T>;
    int const tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q2 = 2 * (lane & 3);
    {  // A's entries start towards L2: a column's 128-byte line per thread
        int const c = tid % kNB, r = 16 * (tid / kNB);
        if (c < nb && r < mr) asm volatile("prefetch.global.L2 [%0];" ::"l"(A + k0 + r0 + r + (int64_t)(k0 + c) * lda));
    }
    int64_t sum[2][2][4];
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[t][n][e] = 0;
    int const slabs = k0 / kNB;
    for (int s = 0; s < slabs; s += 2) {
        int const ns = min(2, slabs - s);
        for (int u = 0; u < ns; ++u) stage_columns<T>(stage, W, ldw, k0, r0, mr, nb, s + u);
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        cta_sync<T>();
        for (int e = tid; e < 64 * ns; e += T) {  // slab u, column n of the product, k = 2 q, 2 q + 1, 2 q + 8, 2 q + 9
            int const u = e >> 6, n = (e >> 2) & 15, q = e & 3;
            int64_t const* src = stage + (u * kNB + 2 * q) * S::RS + (r0 == 0 ? 0 : T) + n;
            uint32_t d0[8], d1[8];
            digit_pairs(d0, src[0], src[S::RS]);
            digit_pairs(d1, src[8 * S::RS], src[9 * S::RS]);
            uint4* dst = digits + (u * 2 + (n >> 3)) * 4 * 32 + (n & 7) * 4 + q;
#pragma unroll
            for (int i = 0; i < 4; ++i) dst[i * 32] = make_uint4(d0[2 * i], d1[2 * i], d0[2 * i + 1], d1[2 * i + 1]);
        }
        cta_sync<T>();
#pragma unroll
        for (int t = 0; t < 2; ++t) {
            int const first = 16 * (warp + S::kWarps * t);
            if (first < mr) {  // warp-uniform
                float acc[2][8][4];
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int e = 0; e < 4; ++e) acc[n][i][e] = 12582912.0f;
#pragma unroll 1
                for (int u = 0; u < ns; ++u) {
                    uint32_t a[8][4];
#pragma unroll
                    for (int h = 0; h < 4; ++h) {  // fragment register h: rows g + 8 (h & 1), k = 2 q + 8 (h >> 1)
                        int64_t const* src = stage + (u * kNB + q2 + 8 * (h >> 1)) * S::RS + first + g + 8 * (h & 1);
                        uint32_t d[8];
                        digit_pairs(d, src[0], src[S::RS]);
#pragma unroll
                        for (int i = 0; i < 8; ++i) a[i][h] = d[i];
                    }
#pragma unroll
                    for (int n = 0; n < 2; ++n) {
                        uint4 const* dig = digits + (u * 2 + n) * 4 * 32 + lane;
#pragma unroll
                        for (int jj = 0; jj < 4; ++jj) {
                            uint4 const v = dig[jj * 32];
#pragma unroll
                            for (int i = 0; i + 2 * jj < 8; ++i) mma_f16(acc[n][i + 2 * jj], a[i], v.x, v.y);
#pragma unroll
                            for (int i = 0; i + 2 * jj + 1 < 8; ++i) mma_f16(acc[n][i + 2 * jj + 1], a[i], v.z, v.w);
                        }
                    }
                }
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        constexpr uint32_t kStart = 0x4b400000u;  // the bits of 1.5 x 2^23
                        int32_t v[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            v[i] = (int32_t)(__float_as_uint(acc[n][2 * i][e]) * 256u +
                                             (__float_as_uint(acc[n][2 * i + 1][e]) - kStart * 257u));
                        int64_t hi = v[1], lo = v[3] + 128;  // units of 2^-38 and 2^-70
                        fix64::mad(hi, v[0], 65536);
                        fix64::mad(lo, v[2], 65536);
                        sum[t][n][e] += (hi << 24) + (lo >> 8);
                    }
            }
        }
        cta_sync<T>();  // the staged columns are written again
    }
#pragma unroll
    for (int t = 0; t < 2; ++t)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int const r = 16 * (warp + S::kWarps * t) + g + 8 * h;
            if (r < mr) {
                int const er = scale[k0 + r0 + r];
                bool ok = true;
#pragma unroll
                for (int n = 0; n < 2; ++n)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        int const c = 8 * n + q2 + e;
                        int64_t v = 0;
                        if (c < nb && r0 + r >= c)
                            ok &= fix64::from_double(A[(k0 + r0 + r) + (int64_t)(k0 + c) * lda], er + scale[k0 + c], v);
                        C[c * S::CS + r] = v - sum[t][n][2 * h + e];
                    }
                if (!ok) atomicOr(row + k0 + r0 + r, fix64::kTodo);
            }
        }
}

// An entry of the workspace.
template <int T>
__device__ __forceinline__ int64_t to_workspace(int64_t q) {
    return Shape<T>::kTensor ? fix64::to_digits(q) : fix64::pack(fix64::split(q));
}
template <int T>
__device__ __forceinline__ int64_t from_workspace(int64_t w) {
    return Shape<T>::kTensor ? fix64::from_digits(w) : fix64::join(fix64::unpack(w));
}

// Why the panels end early: a row, or the whole panel, is left to binary64.
constexpr int kStopRow = 1, kStopPanel = 2;

// A panel from the side of its rows: entry (i, j) is in row k0 + i and column k0 + j.
struct Panel {
    int k0, nb;
    const double* A;  // the matrix from (0, 0) of the panel on
    int64_t lda;
    int64_t* W;       // the workspace's columns from row k0 on
    int64_t ldw;
    const Limbs* D;   // the diagonal block, row by row
    uint32_t* row;    // the rows' words
    uint32_t below;   // fix64::weak_below
    int* stop;
};

// Whether fixed point serves row i although some of its entries in the panel are weak (fix64.cuh). x: those entries,
// CS apart; one thread.
template <int T>
__device__ __forceinline__ bool served(Panel const& p, int i, const int64_t* x, unsigned weak) {
    using S = Shape<T>;
    int const J = p.k0 / kNB, first = fix64::first_panel(p.row[i]);
    unsigned zeros = 0;
    for (; weak != 0 && first <= J; weak &= weak - 1) {
        int const j = __ffs(weak) - 1;
        uint32_t terms = 0;
        bool any = false;
#pragma unroll 1
        for (int k = kNB * max(first, fix64::first_panel(p.row[j])); k < p.k0 && terms < p.below; k += 2) {
            int64_t u[2], v[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) u[c] = p.W[i + (k + c) * p.ldw], v[c] = p.W[j + (k + c) * p.ldw];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                int64_t const a = from_workspace<T>(u[c]), b = from_workspace<T>(v[c]);
                terms += fix64::term(fix64::split(a).h, fix64::split(b).h);
                any |= a != 0 && b != 0;
            }
        }
#pragma unroll 1
        for (int k = 0; k < p.nb && terms < p.below; ++k) {
            if (k == i || k == j) continue;
            Limbs const a = k < i ? fix64::split(x[k * S::CS]) : p.D[k * kNB + i];
            Limbs const b = p.D[max(j, k) * kNB + min(j, k)];
            terms += fix64::term(a.h, b.h);
            any |= k < j && (a.h | a.l) != 0 && (b.h | b.l) != 0;
        }
        if (terms < p.below) {
            if (any || x[j * S::CS] != 0) return false;
            zeros |= 1u << j;
        }
    }
    if ((zeros | weak) == 0) return true;
    bool exact = true;
#pragma unroll 4
    for (int j = 0; j < kNB; ++j)
        if (((zeros | weak) >> j & 1) != 0) exact &= p.A[i + j * p.lda] == 0.0;
    return exact;
}

// What a row's way through the panel leaves.
struct RowState {
    bool ok = true;  // in range
    unsigned weak = 0;  // entries
    int64_t squares = 0;
    int any = 0;
};

// Row i's word after the panel.
__device__ __forceinline__ void note_row(Panel const& p, int i, RowState const& s) {
    p.row[i] = fix64::row_after(p.row[i], p.k0 / kNB, s.squares, s.any != 0);
}

// Whether row i is certified, once its word and the diagonal block's rows' are noted. One thread. Out of line, and as
// few instructions as can be: what is executed once in a while is not in the instruction cache (n = 128 x 4,000, with
// five weak entries a matrix: 1.72 ms, 2.05 when a row with one was gone through entry by entry, 1.51 without a look
// at them).
template <int T>
__device__ __noinline__ bool certified(Panel const p, int i, const int64_t* x, bool in_range, unsigned weak) {
    uint32_t const word = p.row[i];
    return in_range && (word & fix64::kTodo) == 0 && (word & fix64::kNormMask) <= fix64::kNormMost &&
           (weak == 0 || served<T>(p, i, x, weak));
}

// Row i of the panel to the workspace, its first `entries` columns, if it is certified; else it is left to binary64.
template <int T>
__device__ __forceinline__ void store_row(Panel const& p, int i, int entries, const int64_t* x, bool ok) {
    if (!ok) {
        p.row[i] |= fix64::kTodo;
        *p.stop = kStopRow;
        return;
    }
#pragma unroll 4
    for (int j = 0; j < entries; ++j) p.W[i + (p.k0 + j) * p.ldw] = to_workspace<T>(x[j * Shape<T>::CS]);
}

// The panel's first 32 rows (mr of them exist), one warp, a row per lane: the 16 columns right-looking.
// Leaves the diagonal block's entries in D and the pivots' reciprocal square roots in rsq.
template <int T>
__device__ __forceinline__ void factor_diagonal(Panel const& p, int mr, int64_t* C, Limbs* D, Rsqrt* rsq) {
    using S = Shape<T>;
    int const lane = threadIdx.x & 31, nb = p.nb;
    bool const mine = lane < mr;
    int64_t sum[kNB], cross[kNB];
#pragma unroll
    for (int c = 0; c < kNB; ++c) {
        sum[c] = mine && c < nb ? C[c * S::CS + lane] : 0;
        cross[c] = fix64::kCrossOfRemainder;
    }
    bool good = true;
    RowState state;
    // The next pivot's reciprocal square root is taken as soon as its column is up to date, beside the
    // products of the columns after it.
    int64_t t = 0;
    Rsqrt y;
    auto pivot = [&](int c) {
        t = fix64::remainder_of(sum[0], cross[0]);
        int64_t const s = __shfl_sync(0xffffffffu, t, c);
        good &= s >= fix64::kPivotMin || c >= nb;
        y = fix64::pivot_rsqrt(max(s, fix64::kPivotMin));
    };
    pivot(0);
    fix64::triangle(nb, [&](auto left, int j) {
        int64_t q;
        bool const in = fix64::scale_entry(t, y, q);
        Limbs const v = fix64::split(q);
        if (lane >= j) {
            state.ok &= in;
            fix64::add_square(state.squares, v.h);
        }
        if (lane > j) {
            if (fix64::weak(t, p.below)) state.weak |= 1u << j;
            state.any |= v.h | v.l;
        }
        if (mine) C[j * S::CS + lane] = q;
        if (lane < kNB) D[lane * kNB + j] = v;
        if (lane == 0) rsq[j] = y;
#pragma unroll
        for (int u = 1; u < decltype(left)::value; ++u) {
            int const c = j + u;  // past the last column: sums that are not used
            fix64::take_off(sum, cross, u, v, Limbs{__shfl_sync(0xffffffffu, v.l, c), __shfl_sync(0xffffffffu, v.h, c)});
            if (u == 1) pivot(c);
        }
    });
    if (mine) note_row(p, lane, state);
    __syncwarp();
    // The diagonal block's rows are certified before any row is stored.
    bool const ok = mine && certified<T>(p, lane, C + lane, state.ok, state.weak);
    if (__all_sync(0xffffffffu, good && (ok || !mine || lane >= nb))) {
        if (mine) store_row<T>(p, lane, min(lane + 1, nb), C + lane, ok);
    } else if (lane == 0) {
        *p.stop = kStopPanel;
    }
}

// Row i of the panel, r of the chunk, against the diagonal block, one thread.
template <int T>
__device__ __forceinline__ void solve_row(Panel const& p, int i, int r, int64_t* C, const Limbs* D, const Rsqrt* rsq) {
    using S = Shape<T>;
    int64_t sum[kNB], cross[kNB];
#pragma unroll
    for (int c = 0; c < kNB; ++c) {
        sum[c] = C[c * S::CS + r];
        cross[c] = fix64::kCrossOfRemainder;
    }
    RowState state;
    fix64::triangle(kNB, [&](auto left, int j) {
        int64_t q;
        int64_t const t = fix64::remainder_of(sum[0], cross[0]);
        state.ok &= fix64::scale_entry(t, rsq[j], q);
        if (fix64::weak(t, p.below)) state.weak |= 1u << j;
        Limbs const v = fix64::split(q);
        C[j * S::CS + r] = q;
        fix64::add_square(state.squares, v.h);
        state.any |= v.h | v.l;
        Limbs const* d = D + j * (kNB + 1);  // past the last row: what follows D, for sums that are not used
#pragma unroll
        for (int u = 1; u < decltype(left)::value; ++u) fix64::take_off(sum, cross, u, v, d[u * kNB]);
    });
    note_row(p, i, state);
    store_row<T>(p, i, kNB, C + r, certified<T>(p, i, C + r, state.ok, state.weak));
}

// One matrix. W: the fixed-point factor while the matrix is being factored, n rows of 8 bytes per
// column with leading dimension ldw; may be L. L2 (optional): a second copy of the factor.
struct FixItem {
    int n;
    const double* A;
    int64_t lda;
    double* L;
    int64_t ldl;
    double* W;
    int64_t ldw;
    double* L2;
    int64_t ldl2;
};

template <int T, class Batch>
__global__ void __launch_bounds__(T, T == 128 ? 3 : T == 64 ? 7 : 11) potrf_fix_kernel(Batch batch, int32_t* info) {
    using S = Shape<T>;
    extern __shared__ __align__(16) unsigned char smem[];
    int64_t* stage = reinterpret_cast<int64_t*>(smem + S::kStage);
    uint4* digits = reinterpret_cast<uint4*>(smem + S::kDigits);
    int64_t* C = reinterpret_cast<int64_t*>(smem + S::kChunk);
    Limbs* D = reinterpret_cast<Limbs*>(smem + S::kDiag);
    Rsqrt* rsq = reinterpret_cast<Rsqrt*>(smem + S::kRsqrt);
    short* scale = reinterpret_cast<short*>(smem + S::kScale);
    uint32_t* row = reinterpret_cast<uint32_t*>(smem + S::kRow);
    __shared__ int s_stop;
    int64_t const b = blockIdx.x;
    FixItem it;
    if (!batch.get(b, it) || it.n > S::NMAX) return;
    int const n = it.n, tid = threadIdx.x;
    int64_t* W = reinterpret_cast<int64_t*>(it.W);
    if (tid == 0) s_stop = 0;
    cta_sync<T>();
    for (int i = tid; i < n; i += T) {
        int e;
        if (!fix64::scale_exponent(it.A[i + (int64_t)i * it.lda], e)) s_stop = kStopPanel;
        scale[i] = (short)e;
        row[i] = fix64::kNewRow;
    }
    cta_sync<T>();
    uint32_t const below = fix64::weak_below(n);
    int stop = s_stop, k0 = 0, r0 = 0;
    for (; k0 < n && stop == 0; k0 += stop == 0 ? kNB : 0) {
        int const nb = min(kNB, n - k0), m = n - k0;
        Panel const p{k0, nb, it.A + k0 + k0 * it.lda, it.lda, W + k0, it.ldw, D, row + k0, below, &s_stop};
        for (r0 = 0; r0 < m && stop == 0; r0 += stop == 0 ? T : 0) {
            int const mr = min(T, m - r0);
            if constexpr (S::kTensor) {
                update_chunk_mma<T>(k0, r0, mr, nb, it.A, it.lda, W, it.ldw, stage, digits, C, scale, row);
            } else {
#define BLASTGPU_UPDATE(RA) \
    update_chunk_int<T, RA>(k0, r0, mr, nb, it.A, it.lda, W, it.ldw, stage, C, scale, row)
                switch ((mr + S::RT - 1) / S::RT) {
                    case 1: BLASTGPU_UPDATE(1); break;
                    case 2: BLASTGPU_UPDATE(2); break;
                    case 3: BLASTGPU_UPDATE(3); break;
                    default: BLASTGPU_UPDATE(4); break;
                }
#undef BLASTGPU_UPDATE
            }
            cta_sync<T>();
            if (r0 == 0) {
                if (tid < 32) factor_diagonal<T>(p, mr, C, D, rsq);
                cta_sync<T>();
            }
            // Nobody writes kStopPanel from here on, so every thread sees the same side of it.
            if (s_stop != kStopPanel && tid < mr && (r0 > 0 || tid >= 32)) solve_row<T>(p, r0 + tid, tid, C, D, rsq);
            cta_sync<T>();  // C is written again; the panel's columns are read from now on
            stop = s_stop;  // not written again before the next chunk's barriers
        }
    }
    // Fixed point to binary64, a warp per column: all of it, or what was certified.
    int const whole = stop == 0 ? n : k0, columns = stop == kStopRow ? k0 + kNB : whole;
    auto todo = [=](int i) { return i >= k0 + r0 + T || (row[i] & fix64::kTodo) != 0; };  // in columns whole .. columns-1
    int const lane = tid & 31, warp = tid >> 5;
    for (int c = warp; c < columns; c += T / 32) {
        int64_t const* w = W + (int64_t)c * it.ldw;
        double* l = it.L + (int64_t)c * it.ldl;
        for (int i0 = c; i0 < n; i0 += 128) {
            int64_t v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                int const i = i0 + lane + 32 * u;
                v[u] = i < n ? w[i] : 0;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                int const i = i0 + lane + 32 * u;
                if (i < n && (c < whole || !todo(i))) {
                    double const x = fix64::entry_to_double(from_workspace<T>(v[u]), scale[i] - 61);
                    l[i] = x;
                    if (it.L2) it.L2[i + (int64_t)c * it.ldl2] = x;
                }
            }
        }
    }
    int fail = 0;
    if (stop != 0) {
        double* F = it.L2 ? it.L2 : it.L;
        int64_t const ldf = it.L2 ? it.ldl2 : it.ldl;
        auto sync = [] { cta_sync<T>(); };
        sync();
        fail = potrf_strips<T>(n, whole, columns, [=](int r, int c) { return it.A[r + c * it.lda]; },
                               [=](int r, int c) -> double& { return F[r + c * ldf]; }, todo,
                               reinterpret_cast<double*>(rsq), tid, sync);
        for (int c = whole + warp; c < n && it.L2; c += T / 32)
            for (int i = c + lane; i < n; i += 32) it.L[i + (int64_t)c * it.ldl] = it.L2[i + (int64_t)c * it.ldl2];
    }
    if (info && tid == 0) info[b] = fail;
}

struct FixStrided {
    int n;
    const double* A; int lda; int64_t sa;
    double* L; int ldl; int64_t sl;
    double* W; int ldw; int64_t sw;      // nullptr: L
    double* L2; int ldl2; int64_t sl2;   // nullptr: none
    __device__ bool get(int64_t b, FixItem& it) const {
        it.n = n;
        it.A = A + b * sa, it.lda = lda;
        it.L = L + b * sl, it.ldl = ldl;
        it.W = W ? W + b * sw : it.L, it.ldw = W ? ldw : ldl;
        it.L2 = L2 ? L2 + b * sl2 : nullptr, it.ldl2 = ldl2;
        return true;
    }
};

// Ragged batches: descriptors with A and L; instances with fewer than min_n rows, and those without A
// (solves with a given factor), are left to the caller's other kernels.
template <class Desc>
struct FixDesc {
    const Desc* desc;
    int min_n;
    __device__ bool get(int64_t b, FixItem& it) const {
        Desc const& d = desc[b];
        it.n = d.A.rows;
        it.A = d.A.data, it.lda = d.A.ld;
        it.L = d.L.data, it.ldl = d.L.ld;
        it.W = it.L, it.ldw = it.ldl;
        it.L2 = nullptr, it.ldl2 = 0;
        return it.A != nullptr && it.n >= min_n;
    }
};

template <int T, class Batch>
int launch_t(Batch const& batch, int64_t count, int32_t* info, cudaStream_t s) {
    constexpr size_t smem = Shape<T>::kBytes;
    cudaError_t const e = ensure_smem<potrf_fix_kernel<T, Batch>>(smem);
    if (e != cudaSuccess) { set_cuda_error(e); return BLASTGPU_ERR_CUDA; }
    potrf_fix_kernel<T, Batch><<<(unsigned)count, T, smem, s>>>(batch, info);
    return check_launch();
}

template <class Batch>
int launch_n(Batch const& batch, int max_n, int64_t count, int32_t* info, cudaStream_t s) {
    if (count == 0) return BLASTGPU_SUCCESS;
    if (count > 0x7fffffff || max_n > 512) return BLASTGPU_ERR_TOO_LARGE;
    int const t = tune_get_bin("potrf_fix.threads", max_n, max_n <= 64 ? 32 : max_n <= 128 ? 64 : 128);
    if (t <= 32 && max_n <= Shape<32>::NMAX) return launch_t<32>(batch, count, info, s);
    if (t <= 64 && max_n <= Shape<64>::NMAX) return launch_t<64>(batch, count, info, s);
    return launch_t<128>(batch, count, info, s);
}

}  // namespace

int launch_potrf_fix(int n, const double* A, int lda, int64_t sa, double* L, int ldl, int64_t sl, double* W, int ldw,
                     int64_t sw, double* L2, int ldl2, int64_t sl2, int32_t* info, int64_t batch, cudaStream_t s) {
    return launch_n(FixStrided{n, A, lda, sa, L, ldl, sl, W, ldw, sw, L2, ldl2, sl2}, n, batch, info, s);
}

int launch_potrf_fix(const blastgpu_posv_desc* desc, int min_n, int max_n, int32_t* info, int64_t batch,
                     cudaStream_t s) {
    return launch_n(FixDesc<blastgpu_posv_desc>{desc, min_n}, max_n, batch, info, s);
}

int launch_potrf_fix(const blastgpu_posv_bwd_desc* desc, int min_n, int max_n, int32_t* info, int64_t batch,
                     cudaStream_t s) {
    return launch_n(FixDesc<blastgpu_posv_bwd_desc>{desc, min_n}, max_n, batch, info, s);
}

}  // namespace blastgpu
