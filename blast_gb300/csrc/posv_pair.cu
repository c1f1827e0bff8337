// Batched binary64 Cholesky factorisation in 64-bit fixed point (fix64.cuh) and solve, n <= 64, sm_103a:
// two matrices per warp, each in shared memory.
//
// Reference: blast::potrf (dense/Potrf.hpp:66-106), left-looking, and blast::trsm (dense/Trsm.hpp:17-66)
// for the solves.
//
// What bounds it: integer instructions, 30,000 for two matrices of n = 48 without right-hand sides, a
// quarter of them the products of block columns, the chain of pivots, with 8 warps per SM, and fetching
// them (fix64::triangle); then the solves' multiply-adds on the binary64 pipe. 50,000 matrices of n = 48 with 8
// right-hand sides take 3.42 ms (1.41 ms the factor alone) against 4.15 ms for a binary64 thread per
// matrix; 10,000 take a half, one matrix of n = 24 23 us a call instead of 53. A matrix has 16 lanes, so that
// the work on the diagonal, which has 16 rows to share it, fills the warp with two matrices, and a batch of
// small matrices needs few warps. The matrix is read from memory once and written once; the earlier
// columns, which a thread per matrix reads again for every strip, stay in shared memory.
//
// The matrix is cut into 16 x 16 blocks (n rounded up), of which the lower ones are stored, each as 16
// columns of 17 entries of 8 bytes: the matrix's binary64 entry at first, then the remainder, then the
// factor's two limbs. The odd stride keeps reads along rows free of bank conflicts as well, and every
// offset within a block is a constant. Per block column:
//  * block products: lane (rt, ct) of the 16 holds rows rt + 4 i and columns 4 ct + j of a block;
//  * the diagonal block: a row per lane, right-looking in registers, the pivot row's limbs by shuffles;
//  * the blocks below: a row per lane against the diagonal block.
// Each integer sum is exact until it is rounded at the end of these steps, and potrf_fix.cu takes the
// same steps, so the factor is the same bits from both. A matrix whose block column cannot be certified
// (fix64.cuh) has its columns from there on factored in binary64 (potrf_strips.cuh) at the end, by its 16 lanes.
//
// Solves in binary64, up to 8 right-hand sides at a time, from the factor's blocks converted in place: a
// solution's entries may lie any number of binades apart, and a column of the factor has no norm that
// bounds the sums. The binary64 pipe stands idle otherwise.
#include "common.cuh"
#include "fix64.cuh"
#include "potrf_strips.cuh"

namespace blastgpu {
namespace {

using fix64::Limbs;
using fix64::Rsqrt;

constexpr int kB = 16;      // block size
constexpr int kMaxN = 64;
constexpr int kGroup = 8;   // right-hand sides solved together

// Shared memory of one matrix with N block columns, in bytes from its start: 13.5 KB at N = 3, so that eight
// warps fit an SM, two to a scheduler. The reciprocals that the solves need take the place of what follows the
// blocks, and the right-hand sides that of the diagonal blocks' upper triangles (RhsBlock).
struct Layout {
    int rsqrt, scale, row, bytes;
};
constexpr int kS = kB + 1;         // column stride of a block
constexpr int kBlock = kB * kS;    // entries of a block
// First entry of block (I, J), J <= I.
__host__ __device__ __forceinline__ int block_at(int I, int J) { return (I * (I + 1) / 2 + J) * kBlock; }
__host__ __device__ __forceinline__ Layout layout_of(int N) {
    Layout l;
    l.rsqrt = 8 * block_at(N, 0);
    l.scale = l.rsqrt + 16 * kB;
    l.row = l.scale + 4 * kB * N;
    l.bytes = l.rsqrt + max(8 * kB * N, l.row + 4 * kB * N - l.rsqrt);
    return l;
}

// Entry i of right-hand side c (< kGroup) of a block, counted from the first entry of the diagonal block: column 8 + c
// has room for 8 + c entries above its diagonal and one below its last row, column 7 - c for the others.
struct RhsBlock {
    int a, b, split;
    __device__ __forceinline__ explicit RhsBlock(int c) : a((8 + c) * kS), b((7 - c) * kS - 8 - c), split(8 + c) {}
    __device__ __forceinline__ int operator()(int i) const { return i == kB - 1 ? a + kB : (i < split ? a : b) + i; }
};

struct PairItem {
    int n, nrhs;
    const double* A;
    int64_t lda;
    double* L;
    int64_t ldl;
    const double* B;
    int64_t ldb;
    double* X;
    int64_t ldx;
};

// One step of a block product: rows v[RA] against columns w[4].
template <int RA>
__device__ __forceinline__ void product_step(int64_t (&hh)[RA][4], int64_t (&cr)[RA][4], Limbs const (&v)[RA],
                                             Limbs const (&w)[4]) {
#pragma unroll
    for (int i = 0; i < RA; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            fix64::mad(hh[i][j], v[i].h, w[j].h);
            fix64::mad(cr[i][j], v[i].h, w[j].l);
            fix64::mad(cr[i][j], v[i].l, w[j].h);
        }
}

// Block (I, J) of the matrix: binary64 entries to the remainders A - L L^T over the block columns
// before J, for the block's first 4 RA rows. False if an entry is out of range.
template <int RA>
__device__ __forceinline__ bool block_remainder(int64_t* P, int n, int I, int J, const int* scale, int rt, int ct) {
    int64_t* blk = P + block_at(I, J) + 4 * ct * kS + rt;
    int64_t hh[RA][4], cr[RA][4];
    int ec[4];
    bool ok = true;
#pragma unroll
    for (int j = 0; j < 4; ++j) ec[j] = scale[kB * J + 4 * ct + j];
#pragma unroll
    for (int i = 0; i < RA; ++i) {
        int const row = kB * I + rt + 4 * i, er = scale[row];
        int const cols = row < n ? row - kB * J - 4 * ct : -1;  // columns 0 .. cols of this lane's four exist
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int64_t v;
            bool const in = fix64::from_double(__longlong_as_double(blk[j * kS + 4 * i]), er + ec[j], v);
            ok &= in || j > cols;
            hh[i][j] = j <= cols ? -v : 0;
            cr[i][j] = fix64::kCrossStart;
        }
    }
    for (int K = 0; K < J; ++K) {
        int64_t const* rows = P + block_at(I, K) + rt;
        int64_t const* cols = P + block_at(J, K) + 4 * ct;
#pragma unroll 4
        for (int k = 0; k < kB; ++k) {
            Limbs v[RA], w[4];
#pragma unroll
            for (int i = 0; i < RA; ++i) v[i] = fix64::unpack(rows[4 * i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = fix64::unpack(cols[j]);
            product_step<RA>(hh, cr, v, w);
            rows += kS;
            cols += kS;
        }
        if ((K & 1) != 0) {  // fix64::kFold terms since the last time
#pragma unroll
            for (int i = 0; i < RA; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) fix64::fold(hh[i][j], cr[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < RA; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) blk[j * kS + 4 * i] = -fix64::total(hh[i][j], cr[i][j]);
    return ok;
}

// A diagonal block, a row per lane (16 lanes per matrix), right-looking. rows: rows of the block that the matrix
// has; cols: columns that some matrix of the warp has. False if a pivot is too small, or the lane's row out of
// range; what follows is not used then. weak: the row's weak entries (fix64.cuh).
__device__ __forceinline__ bool factor_diagonal(int64_t* blk, int rows, int cols, Rsqrt* rsq, uint32_t& row, int J, int l16,
                                                uint32_t below, unsigned& weak) {
    blk += l16;
    int64_t sum[kB], cross[kB];
#pragma unroll
    for (int c = 0; c < kB; ++c) {
        sum[c] = l16 < cols ? blk[c * kS] : 0;
        cross[c] = fix64::kCrossOfRemainder;
    }
    bool good = true, off = false;
    int64_t squares = 0, t = 0;
    int any = 0;
    Rsqrt y;
    // The next pivot's reciprocal square root is taken as soon as its column is up to date, beside the
    // products of the columns after it.
    auto pivot = [&](int c) {
        t = fix64::remainder_of(sum[0], cross[0]);
        int64_t const s = __shfl_sync(0xffffffffu, t, c, kB);
        good &= s >= fix64::kPivotMin || c >= rows;
        y = fix64::pivot_rsqrt(max(s, fix64::kPivotMin));
    };
    pivot(0);
    fix64::triangle(cols, [&](auto left, int j) {
        int64_t q;
        bool const ok = fix64::scale_entry(t, y, q);
        Limbs const v = fix64::split(q);
        blk[j * kS] = fix64::pack(v);
        if (l16 >= j) {
            off |= !ok;
            fix64::add_square(squares, v.h);
        }
        if (l16 > j) {
            if (fix64::weak(t, below)) weak |= 1u << j;
            any |= v.h | v.l;
        }
        if (l16 == 0) rsq[j] = y;
#pragma unroll
        for (int u = 1; u < decltype(left)::value; ++u) {
            int const c = j + u;  // past the last column: sums that are not used
            fix64::take_off(sum, cross, u, v, Limbs{__shfl_sync(0xffffffffu, v.l, c, kB), __shfl_sync(0xffffffffu, v.h, c, kB)});
            if (u == 1) pivot(c);
        }
    });
    if (l16 >= rows) return good;
    row = fix64::row_after(row, J, squares, any != 0);
    return (row & fix64::kNormMask) <= fix64::kNormMost && good && !off;
}

// A row (this lane's, at x) against the diagonal block D; mine: the row exists (else it becomes zeros). False if
// it is out of range.
__device__ __forceinline__ bool solve_block_row(int64_t* x, bool mine, const int64_t* D, const Rsqrt* rsq, uint32_t& row,
                                                int J, uint32_t below, unsigned& weak) {
    int64_t sum[kB], cross[kB];
#pragma unroll
    for (int c = 0; c < kB; ++c) {
        sum[c] = mine ? x[c * kS] : 0;
        cross[c] = fix64::kCrossOfRemainder;
    }
    bool ok = true;
    int64_t squares = 0;
    int any = 0;
    fix64::triangle(kB, [&](auto left, int j) {
        int64_t q;
        int64_t const t = fix64::remainder_of(sum[0], cross[0]);
        ok &= fix64::scale_entry(t, rsq[j], q);
        if (fix64::weak(t, below)) weak |= 1u << j;
        Limbs const v = fix64::split(q);
        x[j * kS] = fix64::pack(v);
        fix64::add_square(squares, v.h);
        any |= v.h | v.l;
        int64_t const* d = D + j * (kS + 1);
#pragma unroll
        for (int u = 1; u < decltype(left)::value; ++u) fix64::take_off(sum, cross, u, v, fix64::unpack(d[u]));
    });
    row = fix64::row_after(row, J, squares, any != 0);
    return (row & fix64::kNormMask) <= fix64::kNormMost && ok;
}

// Whether fixed point serves row i in block column J although some of its entries are weak (fix64.cuh); a lane's own
// affair. row: the rows' words; A: the matrix, n rows. Out of line, and as few instructions as can be: they are not in the
// instruction cache when they are wanted.
__device__ __noinline__ bool served(const int64_t* P, const uint32_t* row, const double* A, int64_t lda, int n, int i, int J,
                                    uint32_t below, unsigned weak) {
    int const base = kB * J, end = min(n, base + kB), first = fix64::first_panel(row[i]);
    auto entry = [&](int r, int c) { return fix64::unpack(P[block_at(r / kB, c / kB) + c % kB * kS + r % kB]); };
    unsigned zeros = 0;
    for (; weak != 0 && first <= J; weak &= weak - 1) {
        int const j = base + __ffs(weak) - 1;
        uint32_t terms = 0;
        bool any = false;
#pragma unroll 1
        for (int k = kB * min(J, max(first, fix64::first_panel(row[j]))); k < end && terms < below; ++k) {
            if (k == i || k == j) continue;
            Limbs const a = entry(max(i, k), min(i, k)), b = entry(max(j, k), min(j, k));
            terms += fix64::term(a.h, b.h);
            any |= k < j && (a.h | a.l) != 0 && (b.h | b.l) != 0;
        }
        if (terms < below) {
            Limbs const q = entry(i, j);
            if (any || (q.h | q.l) != 0) return false;
            zeros |= 1u << (j - base);
        }
    }
    if ((zeros | weak) == 0) return true;
    bool exact = true;
#pragma unroll 4
    for (int j = 0; j < kB; ++j)
        if (((zeros | weak) >> j & 1) != 0) exact &= A[i + (base + j) * lda] == 0.0;
    return exact;
}

// 1 / d, the same bits for d times a power of two.
__device__ __forceinline__ double pivot_reciprocal(double d) {
    int const hi = __double2hiint(d), field = (hi >> 20) & 0x7ff;
    if (hi < 0x00100000 || field == 0x7ff) return 1.0 / d;  // no normal positive number
    return scalbn(rcp_nr(__hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(d))), 1023 - field);
}

// X(:, g0 .. g0 + nr - 1) of one matrix (16 lanes; the other matrix of the warp runs the same steps). P: the factor
// in binary64, zeros from row n on; rd: the reciprocals of its diagonal. RL lanes side by side take a right-hand
// side each, the others rows of a block of 16, up to 8 sums a lane, kRows rows at a time against the diagonal block. With
// 8 right-hand sides only the triangles of 4 rows leave lanes idle. Whatever RL, every entry's sum takes the other
// rows in the order in which they are solved, so a matrix's solution does not depend on its neighbour's.
template <int RL>
__device__ __forceinline__ void solve_group(PairItem const& it, int g0, int nr, int blocks, int n, double* P,
                                            const double* rd, int l16) {
    constexpr int kRows = RL >= 4 ? 4 : kB / RL;  // rows solved together
    constexpr int RW = kRows * RL / kB;           // of which a lane has this many
    constexpr int kSub = kB / kRows;
    int const r = l16 % RL, first = l16 / RL * RW;
    RhsBlock const y(r);
#pragma unroll
    for (int c = 0; c < RL; ++c)
        for (int J = 0; J < blocks; ++J) {
            int const i = kB * J + l16;
            P[block_at(J, J) + RhsBlock(c)(l16)] = c < nr && i < n ? it.B[i + (int64_t)(g0 + c) * it.ldb] : 0.0;
        }
    __syncwarp();
    for (int I = 0; I < blocks; ++I) {
        double* const D = P + block_at(I, I);
        double acc[kSub][RW];
#pragma unroll
        for (int s = 0; s < kSub; ++s)
#pragma unroll
            for (int w = 0; w < RW; ++w) acc[s][w] = D[y(kRows * s + first + w)];
        for (int K = 0; K < I; ++K) {
            double const* l = P + block_at(I, K) + first;
            double const* yk = P + block_at(K, K);
#pragma unroll 8
            for (int k = 0; k < kB; ++k) {
                double const v = yk[y(k)];
#pragma unroll
                for (int s = 0; s < kSub; ++s)
#pragma unroll
                    for (int w = 0; w < RW; ++w) acc[s][w] = fma(-l[k * kS + kRows * s + w], v, acc[s][w]);
            }
        }
#pragma unroll
        for (int j = 0; j < kB; ++j) {
            int const sj = j / kRows, jj = j % kRows;
            double const v = __shfl_sync(0xffffffffu, acc[sj][jj % RW] * rd[kB * I + j], jj / RW * RL + r, kB);
#pragma unroll
            for (int s = sj; s < kSub; ++s)
#pragma unroll
                for (int w = 0; w < RW; ++w) {
                    if (s == sj && first + w == jj) acc[s][w] = v;
                    else if (s > sj || first + w > jj) acc[s][w] = fma(-D[j * kS + kRows * s + first + w], v, acc[s][w]);
                }
        }
#pragma unroll
        for (int s = 0; s < kSub; ++s)
#pragma unroll
            for (int w = 0; w < RW; ++w)
                if (kB * I + kRows * s + first + w < n) D[y(kRows * s + first + w)] = acc[s][w];
        __syncwarp();
    }
    for (int I = blocks - 1; I >= 0; --I) {
        double* const D = P + block_at(I, I);
        double acc[kSub][RW];
#pragma unroll
        for (int s = 0; s < kSub; ++s)
#pragma unroll
            for (int w = 0; w < RW; ++w) acc[s][w] = D[y(kRows * s + first + w)];
        for (int K = blocks - 1; K > I; --K) {
            double const* l = P + block_at(K, I) + first * kS;
            double const* yk = P + block_at(K, K);
#pragma unroll 8
            for (int k = kB - 1; k >= 0; --k) {
                double const v = yk[y(k)];
#pragma unroll
                for (int s = 0; s < kSub; ++s)
#pragma unroll
                    for (int w = 0; w < RW; ++w) acc[s][w] = fma(-l[(kRows * s + w) * kS + k], v, acc[s][w]);
            }
        }
#pragma unroll
        for (int j = kB - 1; j >= 0; --j) {
            int const sj = j / kRows, jj = j % kRows;
            double const v = __shfl_sync(0xffffffffu, acc[sj][jj % RW] * rd[kB * I + j], jj / RW * RL + r, kB);
#pragma unroll
            for (int s = sj; s >= 0; --s)
#pragma unroll
                for (int w = 0; w < RW; ++w) {
                    if (s == sj && first + w == jj) acc[s][w] = v;
                    else if (s < sj || first + w < jj) acc[s][w] = fma(-D[(kRows * s + first + w) * kS + j], v, acc[s][w]);
                }
        }
#pragma unroll
        for (int s = 0; s < kSub; ++s)
#pragma unroll
            for (int w = 0; w < RW; ++w)
                if (kB * I + kRows * s + first + w < n) D[y(kRows * s + first + w)] = acc[s][w];
        __syncwarp();
    }
    // X in whole lines, 16 lanes along a column (one lane per right-hand side writes 8 bytes to a line: 0.9 ms
    // more for 10,000 matrices with X in host memory).
#pragma unroll
    for (int c = 0; c < RL; ++c)
        for (int J = 0; J < blocks; ++J) {
            int const i = kB * J + l16;
            if (c < nr && i < n) it.X[i + (int64_t)(g0 + c) * it.ldx] = P[block_at(J, J) + RhsBlock(c)(l16)];
        }
    __syncwarp();
}

// Operands in host memory (HOST): the link to it carries lines of 16 entries, and its memory is read and written
// fastest along one stretch. So the columns are read one after another, each in whole lines, and a block column of the
// factor goes out as soon as it is there, with the other direction still busy. 50,000 matrices of n = 48 with 8
// right-hand sides take 4.91 ms with three batches in flight and 5.11 alone (row blocks of A read, and L written,
// at once: 5.25, 5.50), 10,000 1.18 ms (1.29), 30,000 of n = 60 5.2 (5.6); prefetches into L2 gave nothing.
// Columns kB J .. kB J + 15 of the factor:
__device__ __forceinline__ void store_columns(PairItem const& it, int n, int J, const int64_t* P, const int* scale, int l16) {
    for (int col = kB * J; col < min(n, kB * J + kB); ++col) {
        double* l = it.L + (int64_t)col * it.ldl;
        int const at = (int)(reinterpret_cast<uintptr_t>(l) >> 3) & 15;
        for (int r = col - ((col + at) & 15) + l16; r < n; r += kB)
            if (r >= col)
                l[r] = fix64::entry_to_double(fix64::join(fix64::unpack(P[block_at(r / kB, J) + col % kB * kS + r % kB])),
                                              scale[r] - 61);
    }
}

template <bool SOLVE, bool HOST, class Batch>
__global__ void __launch_bounds__(32, 8) posv_pair_kernel(Batch batch, int64_t count, int N, int32_t* info) {
    extern __shared__ __align__(16) unsigned char smem[];
    int const l16 = threadIdx.x & 15, half = threadIdx.x >> 4;
    Layout const lay = layout_of(N);
    unsigned char* base = smem + half * lay.bytes;
    int64_t* P = reinterpret_cast<int64_t*>(base);
    Rsqrt* rsq = reinterpret_cast<Rsqrt*>(base + lay.rsqrt);
    int* scale = reinterpret_cast<int*>(base + lay.scale);
    uint32_t* row = reinterpret_cast<uint32_t*>(base + lay.row);
    int64_t const b = 2 * (int64_t)blockIdx.x + half;
    PairItem it;
    it.n = 0, it.nrhs = 0;
    bool const have = b < count && batch.get(b, it) && it.n <= kB * N;
    int const n = have ? it.n : 0;
    int const nmax = max(n, __shfl_xor_sync(0xffffffffu, n, 16));
    if (nmax == 0) return;
    int const blocks = (nmax + kB - 1) / kB;  // the warp's; the layout stays that of N
    // lower(A) to shared memory, all loads in flight together
    if constexpr (HOST) {
#pragma unroll 2
        for (int j = 0; j < n; ++j) {
            double const* a = it.A + (int64_t)j * it.lda;
            int const at = (int)(reinterpret_cast<uintptr_t>(a) >> 3) & 15;
            for (int r = j - ((j + at) & 15) + l16; r < n; r += kB)
                if (r >= j)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(
                                     P + block_at(r / kB, j / kB) + j % kB * kS + r % kB)), "l"(a + r)
                                 : "memory");
        }
    } else {
        for (int I = 0; I < blocks; ++I) {
            int const r = kB * I + l16;
            if (r < n) {
                for (int J = 0; J <= I; ++J) {
                    unsigned const d = (unsigned)__cvta_generic_to_shared(P + block_at(I, J) + l16);
                    double const* a = it.A + r + (int64_t)(kB * J) * it.lda;
#pragma unroll 4
                    for (int c = 0; c < kB; ++c)
                        if (kB * J + c <= r)
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d + 8 * c * kS), "l"(a + c * it.lda)
                                         : "memory");
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    __syncwarp();
    bool sound = true;  // of this matrix, as far as this lane has seen
    for (int i = l16; i < kB * blocks; i += kB) {
        int e = 0;
        if (i < n) sound &= fix64::scale_exponent(__longlong_as_double(P[block_at(i / kB, i / kB) + i % kB * (kS + 1)]), e);
        scale[i] = e;
        row[i] = fix64::kNewRow;
    }
    unsigned const half_mask = 0xffffu << (16 * half);
    uint32_t const below = fix64::weak_below(n);
    // The first block column that is left to binary64.
    int redo = (__ballot_sync(0xffffffffu, !sound) & half_mask) ? 0 : blocks;
    for (int J = 0; J < blocks && __any_sync(0xffffffffu, n > 0 && redo == blocks); ++J) {
        for (int I = J; I < blocks; ++I) {
            int const rows = nmax - kB * I;  // only the last block can have fewer than 16
            if (rows <= 4) sound &= block_remainder<1>(P, n, I, J, scale, l16 & 3, l16 >> 2);
            else if (rows <= 8) sound &= block_remainder<2>(P, n, I, J, scale, l16 & 3, l16 >> 2);
            else sound &= block_remainder<4>(P, n, I, J, scale, l16 & 3, l16 >> 2);
        }
        __syncwarp();
        auto look = [&](int first, unsigned weak) {
            __syncwarp();
            if (weak != 0 && first + l16 < n && sound && redo == blocks)
                sound = served(P, row, it.A, it.lda, n, first + l16, J, below, weak);
        };
        unsigned weak = 0;
        sound &= factor_diagonal(P + block_at(J, J), min(kB, n - kB * J), min(kB, nmax - kB * J), rsq, row[kB * J + l16], J, l16,
                                 below, weak);
        look(kB * J, weak);
        for (int I = J + 1; I < blocks; ++I) {
            weak = 0;
            sound &= solve_block_row(P + block_at(I, J) + l16, kB * I + l16 < nmax, P + block_at(J, J), rsq, row[kB * I + l16],
                                     J, below, weak);
            look(kB * I, weak);
        }
        __syncwarp();
        if ((__ballot_sync(0xffffffffu, !sound) & half_mask) && redo == blocks) redo = J;
        if constexpr (HOST)
            if (redo == blocks) store_columns(it, n, J, P, scale, l16);
    }
    // The factor becomes binary64 in place and goes to memory; block columns from redo on are read again.
    int fail = 0;
    if (SOLVE || !HOST || __any_sync(0xffffffffu, n > 0 && redo < blocks)) {
        for (int I = 0; I < blocks; ++I) {
            int const r = kB * I + l16, e = scale[r] - 61;
            for (int J = 0; J <= min(I, redo - 1); ++J) {
                int64_t* blk = P + block_at(I, J) + l16;
                double* l = it.L + r + (int64_t)(kB * J) * it.ldl;
#pragma unroll 4
                for (int c = 0; c < kB; ++c) {
                    bool const in = kB * J + c <= r;
                    double const x = fix64::entry_to_double(fix64::join(fix64::unpack(blk[c * kS])), e);
                    if (SOLVE || redo < blocks) blk[c * kS] = in && r < n ? __double_as_longlong(x) : 0;
                    if (!HOST && in && r < n) l[c * it.ldl] = x;
                }
            }
            for (int J = redo; J <= I; ++J)
                for (int c = 0; c < kB; ++c)
                    P[block_at(I, J) + l16 + c * kS] =
                        kB * J + c <= r && r < n ? __double_as_longlong(it.A[r + (int64_t)(kB * J + c) * it.lda]) : 0;
        }
        if (redo < blocks && n > 0) {
            double* F = reinterpret_cast<double*>(P);
            auto at = [=](int r, int c) -> double& { return F[block_at(r / kB, c / kB) + c % kB * kS + r % kB]; };
            auto sync = [=] { __syncwarp(half_mask); };
            sync();
            fail = potrf_strips<kB>(n, kB * redo, 0, at, at, [](int) { return true; }, reinterpret_cast<double*>(rsq), l16, sync);
            for (int c = kB * redo; c < n; ++c)
                for (int r = c / kB * kB + l16; r < n; r += kB)
                    if (r >= c) it.L[r + (int64_t)c * it.ldl] = at(r, c);
        }
    }
    if (info && l16 == 0 && have) info[b] = fail;
    if constexpr (SOLVE) {
        double* F = reinterpret_cast<double*>(P);
        double* rd = reinterpret_cast<double*>(rsq);
        __syncwarp();
        for (int i = l16; i < kB * blocks; i += kB)
            rd[i] = i < n ? pivot_reciprocal(F[block_at(i / kB, i / kB) + i % kB * (kS + 1)]) : 1.0;
        int const nrhs = have ? it.nrhs : 0;
        int const most = max(nrhs, __shfl_xor_sync(0xffffffffu, nrhs, 16));
        for (int g0 = 0; g0 < most; g0 += kGroup) {
            int const nr = max(0, min(kGroup, nrhs - g0)), wide = min(kGroup, most - g0);
            if (wide > 4) solve_group<8>(it, g0, nr, blocks, n, F, rd, l16);
            else if (wide > 2) solve_group<4>(it, g0, nr, blocks, n, F, rd, l16);
            else if (wide == 2) solve_group<2>(it, g0, nr, blocks, n, F, rd, l16);
            else solve_group<1>(it, g0, nr, blocks, n, F, rd, l16);
        }
    }
}

struct PairStrided {
    int n, nrhs;
    const double* A; int lda; int64_t sa;
    double* L; int ldl; int64_t sl;
    const double* B; int ldb; int64_t sb;
    double* X; int ldx; int64_t sx;
    __device__ bool get(int64_t b, PairItem& it) const {
        it = {n, nrhs, A + b * sa, lda, L + b * sl, ldl, B ? B + b * sb : nullptr, ldb, X ? X + b * sx : nullptr, ldx};
        return true;
    }
};

struct PairDesc {
    const blastgpu_posv_desc* desc;
    int min_n;
    __device__ bool get(int64_t b, PairItem& it) const {
        blastgpu_posv_desc const& d = desc[b];
        it = {d.A.rows, d.B.cols, d.A.data, d.A.ld, d.L.data, d.L.ld, d.B.data, d.B.ld, d.X.data, d.X.ld};
        return d.A.data != nullptr && d.A.rows >= min_n;
    }
};

template <bool SOLVE, bool HOST = false, class Batch>
int launch(Batch const& batch, int max_n, int64_t count, int32_t* info, cudaStream_t s) {
    if (count == 0) return BLASTGPU_SUCCESS;
    if (max_n > kMaxN || (count + 1) / 2 > 0x7fffffff) return BLASTGPU_ERR_TOO_LARGE;
    int const N = (max_n + kB - 1) / kB;
    size_t const smem = 2 * (size_t)layout_of(N).bytes;
    cudaError_t const e = ensure_smem<posv_pair_kernel<SOLVE, HOST, Batch>>(2 * (size_t)layout_of(kMaxN / kB).bytes);
    if (e != cudaSuccess) { set_cuda_error(e); return BLASTGPU_ERR_CUDA; }
    posv_pair_kernel<SOLVE, HOST, Batch><<<(unsigned)((count + 1) / 2), 32, smem, s>>>(batch, count, N, info);
    return check_launch();
}

}  // namespace

int launch_posv_pair(int n, int nrhs, const double* A, int lda, int64_t sa, double* L, int ldl, int64_t sl,
                     const double* B, int ldb, int64_t sb, double* X, int ldx, int64_t sx, int32_t* info, int64_t batch,
                     bool host, cudaStream_t s) {
    PairStrided const p{n, nrhs, A, lda, sa, L, ldl, sl, nrhs ? B : nullptr, ldb, sb, nrhs ? X : nullptr, ldx, sx};
    if (host) return nrhs ? launch<true, true>(p, n, batch, info, s) : launch<false, true>(p, n, batch, info, s);
    return nrhs ? launch<true>(p, n, batch, info, s) : launch<false>(p, n, batch, info, s);
}

int launch_posv_pair(const blastgpu_posv_desc* desc, int min_n, int max_n, int32_t* info, int64_t batch, cudaStream_t s) {
    return launch<true>(PairDesc{desc, min_n}, max_n, batch, info, s);
}

}  // namespace blastgpu
