// Batched binary64 Cholesky factorisation and solve in 64-bit fixed point (fix64.cuh), n <= 64, sm_103a:
// two matrices per warp, each in shared memory.
//
// Reference: blast::potrf (dense/Potrf.hpp:66-106), left-looking, and blast::trsm (dense/Trsm.hpp:17-66)
// for the solves.
//
// What bounds it: integer instructions, 28,000 for two matrices of n = 48 without right-hand sides, a
// quarter of them the products of block columns, and the chain of pivots, with 8 warps per SM. 50,000
// matrices of n = 48 with 8 right-hand sides take 3.11 ms (1.24 ms the factor alone) against 4.15 ms for
// a binary64 thread per matrix, which the binary64 pipe holds at 3.0 ms at best; 10,000 take a half, one
// matrix of n = 24 21 us a call instead of 53. A matrix has 16 lanes, so that the work on the diagonal,
// which has 16 rows to share it, fills the warp with two matrices, and a batch of small matrices needs few
// warps. The matrix is read from memory
// once and written once; the earlier columns, which a thread per matrix reads again for every strip,
// stay in shared memory.
//
// The matrix is cut into 16 x 16 blocks (n rounded up), of which the lower ones are stored, each as 16
// columns of 17 entries of 8 bytes: the matrix's binary64 entry at first, then the remainder, then the
// factor's two limbs. The odd stride keeps reads along rows free of bank conflicts as well, and every
// offset within a block is a constant. Per block column:
//  * block products: lane (rt, ct) of the 16 holds rows rt + 4 i and columns 4 ct + j of a block;
//  * the diagonal block: a row per lane, right-looking in registers, the pivot row's limbs by shuffles;
//  * the blocks below: a row per lane against the diagonal block.
// Each integer sum is exact until it is rounded at the end of these steps, and potrf_fix.cu takes the
// same steps, so the factor is the same bits from both.
//
// Solves, 8 right-hand sides at a time: a right-hand side is a row that follows the same steps (y is
// the row b^T L^-T), with an exponent of its own for each block of 16 entries, since nothing bounds a
// solution as the diagonal bounds the factor. A block's entries are first scaled to leave 3 bits for
// growth; should the triangle of the block need more, the block is solved again with 3 bits more.
#include "common.cuh"
#include "fix64.cuh"

namespace blastgpu {
namespace {

using fix64::Limbs;
using fix64::Rsqrt;

constexpr int kB = 16;      // block size
constexpr int kMaxN = 64;
constexpr int kGroup = 8;   // right-hand sides solved together
constexpr int kFwdBits = 60, kBwdBits = 57;  // rows of L have norm < 1/2, its columns only entries < 1/2

// Shared memory of one matrix with N block columns, in bytes from its start.
struct Layout {
    int rsqrt, scale, bad, rhs, expo, bytes;
};
constexpr int kS = kB + 1;         // column stride of a block
constexpr int kBlock = kB * kS;    // entries of a block
// First entry of block (I, J), J <= I.
__host__ __device__ __forceinline__ int block_at(int I, int J) { return (I * (I + 1) / 2 + J) * kBlock; }
__host__ __device__ __forceinline__ Layout layout_of(int N, bool solve) {
    Layout l;
    l.rsqrt = 8 * block_at(N, 0);
    l.scale = l.rsqrt + 16 * kB * N;
    l.bad = l.scale + 4 * kB * N;
    l.rhs = l.bad + kB * N;
    l.expo = l.rhs + (solve ? 8 * kB * kGroup * N : 0);
    l.bytes = (l.expo + (solve ? 4 * kGroup * (N + 1) : 0) + 15) & ~15;
    return l;
}

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
// before J, for the block's first 4 RA rows.
template <int RA>
__device__ __forceinline__ void block_remainder(int64_t* P, int n, int I, int J, const int* scale, unsigned char* bad,
                                                int rt, int ct) {
    int64_t* blk = P + block_at(I, J) + 4 * ct * kS + rt;
    int64_t hh[RA][4], cr[RA][4];
    int ec[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) ec[j] = scale[kB * J + 4 * ct + j];
#pragma unroll
    for (int i = 0; i < RA; ++i) {
        int const row = kB * I + rt + 4 * i, er = scale[row];
        int const cols = row < n ? row - kB * J - 4 * ct : -1;  // columns 0 .. cols of this lane's four exist
        bool ok = true;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            int64_t v;
            bool const in = fix64::from_double(__longlong_as_double(blk[j * kS + 4 * i]), er + ec[j], v);
            ok &= in || j > cols;
            hh[i][j] = j <= cols ? -v : 0;
            cr[i][j] = fix64::kCrossStart;
        }
        if (!ok) bad[row] = fix64::kNoPivot | fix64::kOutOfRange;
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
}

// A diagonal block, a row per lane (16 lanes per matrix), right-looking. fail: the first column whose pivot
// is not positive (unchanged if there is none); what follows it is not used. first: the block's first
// column; cols: columns of the block that some matrix of the warp has.
__device__ __forceinline__ void factor_diagonal(int64_t* blk, int first, int cols, Rsqrt* rsq, unsigned char* bad, int l16,
                                                int& fail) {
    blk += l16;
    int64_t acc[kB], cr[kB];
#pragma unroll
    for (int c = 0; c < kB; ++c) {
        acc[c] = l16 < cols ? blk[c * kS] : 0;
        cr[c] = -fix64::kCrossStart;
    }
    bool const no_pivot = bad[l16] != 0;
    bool off = false;
    // The next pivot's reciprocal square root is taken as soon as its column is up to date, beside the
    // products of the columns after it.
    int64_t t = 0;
    Rsqrt y;
    auto pivot = [&](int c) {
        t = acc[c] - fix64::total(0, -cr[c]);
        int64_t s = __shfl_sync(0xffffffffu, off || no_pivot ? (int64_t)-1 : t, c, kB);
        if (s < fix64::kPivotMin) {
            fail = min(fail, first + c);
            s = int64_t(1) << 60;
        }
        y = fix64::pivot_rsqrt(s);
    };
    pivot(0);
#pragma unroll
    for (int j = 0; j < kB; ++j) {
        if (j < cols) {
            int64_t q;
            bool const ok = fix64::scale_entry<fix64::kEntryBits>(t, y, q);
            off |= !ok && l16 > j;
            Limbs const v = fix64::split(q);
            blk[j * kS] = fix64::pack(v);
            if (l16 == 0) rsq[j] = y;
            int const nh = -v.h, nl = -v.l;
#pragma unroll
            for (int c = j + 1; c < kB; ++c) {
                int const h = __shfl_sync(0xffffffffu, v.h, c, kB), l = __shfl_sync(0xffffffffu, v.l, c, kB);
                fix64::mad(acc[c], nh, h);
                fix64::mad(cr[c], nh, l);
                fix64::mad(cr[c], nl, h);
                if (c == j + 1) pivot(c);
            }
        }
    }
    if (off) bad[l16] = fix64::kNoPivot | fix64::kOutOfRange;
}

// A row (this lane's, at row) against the diagonal block D; mine: the row exists (else it becomes zeros).
__device__ __forceinline__ bool solve_block_row(int64_t* row, bool mine, const int64_t* D, const Rsqrt* rsq) {
    Limbs x[kB];
    bool ok = true;
#pragma unroll
    for (int j = 0; j < kB; ++j) {
        int64_t hh = 0, c0 = fix64::kCrossStart, c1 = 0;
#pragma unroll
        for (int q = 0; q < j; ++q) {
            Limbs const d = fix64::unpack(D[q * kS + j]);
            fix64::mad(hh, x[q].h, d.h);
            fix64::mad(c0, x[q].h, d.l);
            fix64::mad(c1, x[q].l, d.h);
        }
        int64_t v;
        ok &= fix64::scale_entry<fix64::kEntryBits>((mine ? row[j * kS] : 0) - fix64::total(hh, c0 + c1), rsq[j], v);
        x[j] = fix64::split(v);
        row[j * kS] = fix64::pack(x[j]);
    }
    return ok;
}

// Right-hand sides r = rt + 4 i of block J: the remainders at Y (columns of the block, kGroup right-hand
// sides each) take minus the products with the blocks solved so far, forward L(J, K) y_K for K < J,
// backward L(I, J)^T x_I for I > J. expo[K][r]: the solved blocks' exponents, expo[N][r] that of block J.
template <int RA, bool BACK>
__device__ __forceinline__ void rhs_remainder(const int64_t* P, int64_t* Y, const int* expo, int N, int blocks, int J, int rt,
                                              int ct) {
    int64_t acc[RA][4];
    int ez[RA];
#pragma unroll
    for (int i = 0; i < RA; ++i) {
        ez[i] = expo[N * kGroup + rt + 4 * i];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;
    }
    for (int K = BACK ? J + 1 : 0; K < (BACK ? blocks : J); ++K) {
        int64_t const* cols = BACK ? P + block_at(K, J) + 4 * ct * kS : P + block_at(J, K) + 4 * ct;
        int64_t const* rows = Y + K * kB * kGroup + rt;
        int64_t hh[RA][4], cr[RA][4];
#pragma unroll
        for (int i = 0; i < RA; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                hh[i][j] = 0;
                cr[i][j] = fix64::kCrossStart;
            }
#pragma unroll 4
        for (int k = 0; k < kB; ++k) {
            Limbs v[RA], w[4];
#pragma unroll
            for (int i = 0; i < RA; ++i) v[i] = fix64::unpack(rows[4 * i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = fix64::unpack(cols[BACK ? j * kS : j]);
            product_step<RA>(hh, cr, v, w);
            rows += kGroup;
            cols += BACK ? 1 : kS;
        }
#pragma unroll
        for (int i = 0; i < RA; ++i) {
            int const d = min(63, ez[i] - expo[K * kGroup + rt + 4 * i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] += fix64::total(hh[i][j], cr[i][j]) >> d;
        }
    }
#pragma unroll
    for (int i = 0; i < RA; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) (Y[(J * kB + 4 * ct + j) * kGroup + rt + 4 * i]) -= acc[i][j];
}

// One right-hand side of block J (its remainders at y, units of 2^(ez - 62)) against the diagonal block:
// the solution's limbs in place. Returns its exponent.
template <bool BACK>
__device__ __forceinline__ int solve_rhs_block(const int64_t* D, const Rsqrt* rsq, int64_t* y, int ez, int cols) {
    constexpr int kBits = BACK ? kBwdBits : kFwdBits;
    int64_t top = 0;
#pragma unroll
    for (int j = 0; j < kB; ++j) {
        int64_t const z = y[j * kGroup];
        top |= z < 0 ? -z : z;
    }
    int shift = (64 - fix64::clz64((uint64_t)top)) - (kBits - 3);
    for (;;) {
        asm volatile("" ::: "memory");  // the triangle is read again by a second attempt, not kept in registers
        Limbs x[kB];
        bool ok = true;
#pragma unroll
        for (int k = 0; k < kB; ++k) {
            int const j = BACK ? kB - 1 - k : k;
            x[j] = Limbs{0, 0};
            if (j >= cols) continue;  // uniform in the warp
            int64_t hh = 0, c0 = fix64::kCrossStart, c1 = 0;
#pragma unroll
            for (int m = 0; m < k; ++m) {
                int const q = BACK ? kB - 1 - m : m;
                Limbs const d = fix64::unpack(BACK ? D[j * kS + q] : D[q * kS + j]);
                fix64::mad(hh, x[q].h, d.h);
                fix64::mad(c0, x[q].h, d.l);
                fix64::mad(c1, x[q].l, d.h);
            }
            int64_t const z = y[j * kGroup], zs = shift > 0 ? z >> min(shift, 63) : z << -shift;
            int64_t v;
            ok &= fix64::scale_entry<kBits>(zs - fix64::total(hh, c0 + c1), rsq[j], v);
            x[j] = fix64::split(v);
        }
        if (ok || shift > 200) {
#pragma unroll
            for (int j = 0; j < kB; ++j) y[j * kGroup] = fix64::pack(x[j]);
            return ez + shift;
        }
        shift += 3;
    }
}

// X(:, g0 .. g0 + nr - 1) of one matrix (16 lanes; the other matrix of the warp runs the same steps).
template <int RA>
__device__ __forceinline__ void solve_group(PairItem const& it, int g0, int nr, int N, int blocks, int nmax, int n, bool good, const int64_t* P,
                                            const Rsqrt* rsq, const int* scale, int64_t* Y, int* expo, int l16) {
    int const rt = l16 & 3, ct = l16 >> 2;
    bool const mine = l16 < nr;  // this lane's right-hand side
    int const r = l16 & (kGroup - 1);
    int top = -100000;  // largest exponent of the solved blocks
    bool finite = true;
    for (int J = 0; J < blocks; ++J) {
        int64_t* y = Y + J * kB * kGroup;
        int const cols = min(kB, nmax - kB * J);
        int ez = 0;
        if (l16 < kGroup) {
            double b[kB];
            int eb = -100000;
#pragma unroll
            for (int j = 0; j < kB; ++j) {
                int const i = kB * J + j;
                b[j] = mine && i < n ? it.B[i + (int64_t)(g0 + r) * it.ldb] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < kB; ++j) {
                int const field = (__double2hiint(b[j]) >> 20) & 0x7ff;
                finite &= field != 0x7ff;
                int const e = b[j] == 0.0 ? -100000 : max(field, 1) - 1022 - scale[kB * J + j];
                eb = max(eb, e);
            }
            ez = max(eb, top) + 2;
#pragma unroll
            for (int j = 0; j < kB; ++j) {
                int64_t v;
                fix64::from_double(b[j], scale[kB * J + j] + ez, v);
                (y[j * kGroup + r]) = v;
            }
            expo[N * kGroup + r] = ez;
        }
        __syncwarp();
        if (J > 0) {
            rhs_remainder<RA, false>(P, Y, expo, N, blocks, J, rt, ct);
            __syncwarp();
        }
        if (l16 < kGroup) {
            int const e = solve_rhs_block<false>(P + block_at(J, J), rsq + kB * J, y + r, ez, cols);
            expo[J * kGroup + r] = e;
            top = max(top, e);
        }
        __syncwarp();
    }
    top = -100000;
    for (int J = blocks - 1; J >= 0; --J) {
        int64_t* y = Y + J * kB * kGroup;
        int const cols = min(kB, nmax - kB * J);
        int ez = 0;
        if (l16 < kGroup) {
            int const ey = expo[J * kGroup + r];
            ez = max(ey, top) + 2;
            int const d = min(63, ez - ey - 1);
#pragma unroll
            for (int j = 0; j < kB; ++j) (y[j * kGroup + r]) = fix64::join(fix64::unpack(y[j * kGroup + r])) >> d;
            expo[N * kGroup + r] = ez;
        }
        __syncwarp();
        if (J + 1 < blocks) {
            rhs_remainder<RA, true>(P, Y, expo, N, blocks, J, rt, ct);
            __syncwarp();
        }
        if (l16 < kGroup) {
            int const e = solve_rhs_block<true>(P + block_at(J, J), rsq + kB * J, y + r, ez, cols);
            expo[J * kGroup + r] = e;
            top = max(top, e);
        }
        __syncwarp();
    }
    // X in whole lines, 16 lanes along a column (one lane per right-hand side writes 8 bytes to a line: 0.9 ms
    // more for 10,000 matrices with X in host memory).
#pragma unroll
    for (int c = 0; c < kGroup; ++c) {
        bool const ok = __shfl_sync(0xffffffffu, finite, c, kB) && good;
        if (c < nr) {
            for (int J = 0; J < blocks; ++J) {
                int const i = kB * J + l16;
                if (i < n) {
                    double const x = fix64::to_double(fix64::join(fix64::unpack(Y[i * kGroup + c])), expo[J * kGroup + c] - 61 - scale[i]);
                    it.X[i + (int64_t)(g0 + c) * it.ldx] = ok ? x : __longlong_as_double(0x7ff8000000000000ll);
                }
            }
        }
    }
    __syncwarp();
}

// Operands in host memory (HOST): the link to it carries lines of 16 entries, and its memory is read and written
// fastest along one stretch. So the columns are read one after another, each in whole lines, and a block column of the
// factor goes out as soon as it is there, with the other direction still busy. 50,000 matrices of n = 48 with 8
// right-hand sides take 4.91 ms with three batches in flight and 5.11 alone (row blocks of A read, and L written,
// at once: 5.25, 5.50), 10,000 1.18 ms (1.29), 30,000 of n = 60 5.2 (5.6); prefetches into L2 gave nothing.
// Columns kB J .. kB J + 15 of the factor:
__device__ __forceinline__ void store_columns(PairItem const& it, int n, int J, int blocks, int fail, const int64_t* P,
                                              const int* scale, const unsigned char* bad, int l16) {
    for (int col = kB * J; col < min(n, kB * J + kB); ++col) {
        double* l = it.L + (int64_t)col * it.ldl;
        int const at = (int)(reinterpret_cast<uintptr_t>(l) >> 3) & 15;
        for (int r = col - ((col + at) & 15) + l16; r < n; r += kB) {
            if (r < col) continue;
            double const x = fix64::entry_to_double(
                fix64::join(fix64::unpack(P[block_at(r / kB, J) + col % kB * kS + r % kB])), scale[r] - 61);
            int const first_nan = (bad[r] & fix64::kOutOfRange) ? 0 : fail;
            l[r] = col >= first_nan ? __longlong_as_double(0x7ff8000000000000ll) : x;
        }
    }
}

template <bool SOLVE, bool HOST, class Batch>
__global__ void __launch_bounds__(32, 12) posv_pair_kernel(Batch batch, int64_t count, int N, int32_t* info) {
    extern __shared__ __align__(16) unsigned char smem[];
    int const l16 = threadIdx.x & 15, half = threadIdx.x >> 4;
    Layout const lay = layout_of(N, SOLVE);
    unsigned char* base = smem + half * lay.bytes;
    int64_t* P = reinterpret_cast<int64_t*>(base);
    Rsqrt* rsq = reinterpret_cast<Rsqrt*>(base + lay.rsqrt);
    int* scale = reinterpret_cast<int*>(base + lay.scale);
    unsigned char* bad = base + lay.bad;
    int64_t* Y = reinterpret_cast<int64_t*>(base + lay.rhs);
    int* expo = reinterpret_cast<int*>(base + lay.expo);
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
    for (int i = l16; i < kB * blocks; i += kB) {
        int e = 0;
        bool ok = true;
        int const J = i / kB;
        if (i < n)
            ok = fix64::scale_exponent(
                __longlong_as_double(P[block_at(J, J) + (i - kB * J) * (kS + 1)]), e);
        scale[i] = e;
        bad[i] = ok ? 0 : fix64::kNoPivot;
    }
    __syncwarp();
    for (int i = l16; i < n; i += kB) {
        if (bad[i]) {
            int e = scale[i];
            for (int j = 0; j < i; ++j) {
                double const a = __longlong_as_double(P[block_at(i / kB, j / kB) + j % kB * kS + i % kB]);
                if (!bad[j]) e = max(e, fix64::exponent_of(a) - scale[j] + fix64::kGrowth);
            }
            scale[i] = e;
        }
    }
    __syncwarp();
    int fail = n;
    for (int J = 0; J < blocks; ++J) {
        for (int I = J; I < blocks; ++I) {
            int const rows = nmax - kB * I;  // only the last block can have fewer than 16
            if (rows <= 4) block_remainder<1>(P, n, I, J, scale, bad, l16 & 3, l16 >> 2);
            else if (rows <= 8) block_remainder<2>(P, n, I, J, scale, bad, l16 & 3, l16 >> 2);
            else block_remainder<4>(P, n, I, J, scale, bad, l16 & 3, l16 >> 2);
        }
        __syncwarp();
        factor_diagonal(P + block_at(J, J), kB * J, min(kB, nmax - kB * J), rsq + kB * J, bad + kB * J, l16, fail);
        __syncwarp();
        for (int I = J + 1; I < blocks; ++I)
            if (!solve_block_row(P + block_at(I, J) + l16, kB * I + l16 < nmax, P + block_at(J, J), rsq + kB * J)) bad[kB * I + l16] = fix64::kNoPivot | fix64::kOutOfRange;
        __syncwarp();
        if constexpr (HOST) store_columns(it, n, J, blocks, fail, P, scale, bad, l16);
    }
    if (info && l16 == 0 && have) info[b] = fail < n ? fail + 1 : 0;
    // The factor to memory. After a pivot that is not positive the columns from it on are NaN, and so are
    // the rows whose entries left the fixed-point range.
    bool again = !HOST;  // in host memory already, but for rows found out of range since
    if constexpr (HOST)
        for (int i = l16; i < n; i += kB) again |= (bad[i] & fix64::kOutOfRange) != 0;
    again = __any_sync(0xffffffffu, again);
    for (int I = 0; I < (again ? blocks : 0); ++I) {
        int const r = kB * I + l16, e = scale[r] - 61, first_nan = (bad[r] & fix64::kOutOfRange) ? 0 : fail;
        if (r < n) {
            for (int J = 0; J <= I; ++J) {
                int64_t const* blk = P + block_at(I, J) + l16;
                double* l = it.L + r + (int64_t)(kB * J) * it.ldl;
#pragma unroll 4
                for (int c = 0; c < kB; ++c) {
                    int const col = kB * J + c;
                    double const x = fix64::entry_to_double(fix64::join(fix64::unpack(blk[c * kS])), e);
                    if (col <= r) l[c * it.ldl] = col >= first_nan ? __longlong_as_double(0x7ff8000000000000ll) : x;
                }
            }
        }
    }
    if constexpr (SOLVE) {
        // rows past n: their remainders are 0, and so are the solutions' entries; the pivots must exist
        for (int i = n + l16; i < kB * blocks; i += kB) rsq[i] = Rsqrt{0, int32_t(1) << 30, 0, int32_t(1) << 29};
        __syncwarp();
        int const nrhs = have ? it.nrhs : 0;
        int const most = max(nrhs, __shfl_xor_sync(0xffffffffu, nrhs, 16));
        for (int g0 = 0; g0 < most; g0 += kGroup) {
            int const nr = max(0, min(kGroup, nrhs - g0));
            if (min(kGroup, most - g0) <= 4) solve_group<1>(it, g0, nr, N, blocks, nmax, n, fail == n, P, rsq, scale, Y, expo, l16);
            else solve_group<2>(it, g0, nr, N, blocks, nmax, n, fail == n, P, rsq, scale, Y, expo, l16);
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
    size_t const smem = 2 * (size_t)layout_of(N, SOLVE).bytes;
    cudaError_t const e = ensure_smem<posv_pair_kernel<SOLVE, HOST, Batch>>(2 * (size_t)layout_of(kMaxN / kB, SOLVE).bytes);
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
