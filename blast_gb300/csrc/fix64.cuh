// 64-bit fixed-point arithmetic for Cholesky factorisations on the integer multiply pipe.
//
// A product of two 60-bit fixed-point numbers takes three 32 x 32-bit multiplications, each with a 64-bit
// addition. A register-blocked loop of them, operands from shared memory, runs at 8.7 products a clock and
// SM on GB300 (two warps per scheduler); binary64 multiply-adds run at 2, whatever the loop, and on another
// pipe. So a dot product takes a quarter of its binary64 time.
//
// A Cholesky factor suits fixed point. With s_i = sqrt(a_ii), row i of L has 2-norm s_i, so nothing
// in the factorisation of a positive definite matrix grows beyond s_i s_j. Row i is scaled by a
// power of two, 2^-e_i, that brings a_ii into [1/16, 1/4); then every |l_ij| < 1/2, and every partial
// sum of products of two rows is below 1/4 (Cauchy-Schwarz). The scaling follows any power-of-two
// scaling of the unknowns, so the error does not depend on their units.
//
//  * A factor entry is q = l * 2^61 held as q = h * 2^30 + l, two signed 32-bit limbs with
//    |h| <= 2^30 and |l| <= 2^29: 60 bits relative to the row's norm, where binary64 has 53.
//  * A dot product of two rows keeps sum(h h) in units of 2^-62 and sum(h l + l h) in units of 2^-92, both
//    in 64 bits. Both rows' norms are below 1/2, so |sum(h h)| <= 2^60 for any length; the cross sum is at
//    most 2^60 sqrt(length), so it is folded into the other one every 32 terms. The l l products (below
//    2^-64 each) are left out. Columns of a factor and right-hand sides have no such norm: the
//    substitutions are not done in this arithmetic.
//  * A term of the matrix or a remainder is an int64 in units of 2^-62.
//
// Errors: an entry is rounded to 2^-61 and a dot product of k terms adds about sqrt(k) * 2^-62, where
// binary64 rounds every partial sum to 2^-53 of its size.
//
// That is an error of 2^-61 or so of s_i s_j, whatever the sizes of the terms of entry (i, j), while
// binary64's follows them down. Where unknowns are coupled weakly (a kernel's far points, blocks with a
// small entry between them), the solution's small entries come from such small terms. So the kernels
// certify what they factor here, panel by panel, and leave the rest of a matrix to binary64 where
//  * an entry is weak, |l_ij l_jj| below a threshold (weak()), and so is the sum of its other terms |l_ik l_jk|,
//    together with |l_ik l_kj| over the panel's other unknowns, through which i and j are coupled and
//    binary64's errors reach the same unknowns. An entry of zero with no term at all is exact. The
//    threshold is 2^-16 at n = 17 and falls with n, so that the error is at most about 10 n 2^-52 of the
//    terms (weak_shift()). Gaussian and Riccati matrices have no such entry in thousands, and one or two
//    weak entries to look at from n = 48 on;
//  * a pivot is below 2^-42 of its diagonal entry or so (kPivotMin): whether it is positive is then for
//    binary64's own rounding to say;
//  * a row has an entry out of range, or entries whose squares exceed its diagonal entry (kNormMost): the
//    matrix is not positive definite, and sums might wrap;
//  * a diagonal entry is zero, negative or not finite.
#pragma once

#include <stdint.h>

#ifdef __CUDACC__
#define FIX64_FN __host__ __device__ __forceinline__
#else
#define FIX64_FN inline
#endif

namespace blastgpu {
namespace fix64 {

struct Limbs {
    int32_t l, h;  // q = h * 2^30 + l
};

// Factor entries of a positive definite matrix stay below 2^60. (2^32 less is asked for, so that a high limb is
// below 2^30.)
constexpr int64_t kEntryMost = (int64_t(1) << 60) - (int64_t(1) << 32);
// Terms after which the cross sum is folded.
constexpr int kFold = 32;

FIX64_FN int clz64(uint64_t a) {
#ifdef __CUDA_ARCH__
    return __clzll((long long)a);
#else
    return a ? __builtin_clzll(a) : 64;
#endif
}

FIX64_FN uint64_t bits_of(double a) {
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(a);
#else
    uint64_t u;
    __builtin_memcpy(&u, &a, 8);
    return u;
#endif
}

// High words of 32 x 32 products and 32-bit windows of 64 bits.
FIX64_FN uint32_t umul_hi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
FIX64_FN uint32_t lo32(int64_t a) { return (uint32_t)a; }
FIX64_FN int32_t hi32(int64_t a) { return (int32_t)(a >> 32); }

FIX64_FN float approx_rsqrt(float a) {
#ifdef __CUDA_ARCH__
    return rsqrtf(a);
#else
    return 1.0f / __builtin_sqrtf(a);
#endif
}

// a += x * y, 32 x 32 + 64 bits. As plain C++ the signs cost instructions of their own: the loop above took
// 1.55 instead of 0.75 ms.
FIX64_FN void mad(int64_t& a, int32_t x, int32_t y) {
#ifdef __CUDA_ARCH__
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a) : "r"(x), "r"(y));
#else
    a += (int64_t)x * y;
#endif
}

// d = c + x * y.
FIX64_FN void mad_to(int64_t& d, int64_t c, int32_t x, int32_t y) {
#ifdef __CUDA_ARCH__
    asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(d) : "r"(x), "r"(y), "l"(c));
#else
    d = c + (int64_t)x * y;
#endif
}

FIX64_FN Limbs split(int64_t q) {
    int32_t const h = (int32_t)((q + (int64_t(1) << 29)) >> 30);
    return {(int32_t)(lo32(q) - ((uint32_t)h << 30)), h};
}

// Sums of a triangle of 16 columns that a row is taken through, column by column: sum[u], cross[u] belong to the u-th
// column from the one at hand. The remainder of the first, once it is up to date:
FIX64_FN int64_t remainder_of(int64_t sum, int64_t cross) { return sum - ((-cross) >> 30); }
constexpr int64_t kCrossOfRemainder = -(int64_t(1) << 29);
// Takes the product of the entry v of the column at hand with d off column u and moves its sums on.
template <int N>
FIX64_FN void take_off(int64_t (&sum)[N], int64_t (&cross)[N], int u, Limbs v, Limbs d) {
    mad_to(sum[u - 1], sum[u], -v.h, d.h);
    mad_to(cross[u - 1], cross[u], -v.h, d.l);
    mad(cross[u - 1], -v.l, d.h);
}

#ifdef __CUDACC__
// Runs column() for the 16 columns of a triangle, up to `cols` of them: its argument is how many columns are left, as a
// type, rounded up to 16, 12, 8 or 4. The four loops are not unrolled: all 16 columns one after another were 56 KB of
// code, and the kernels' warps waited for the instruction cache.
template <int LEFT>
struct Left {
    static constexpr int value = LEFT;
};
template <class Column>
__device__ __forceinline__ void triangle(int cols, Column&& column) {
    int j = 0;
#pragma unroll 1
    for (; j < min(4, cols); ++j) column(Left<16>{}, j);
#pragma unroll 1
    for (; j < min(8, cols); ++j) column(Left<12>{}, j);
#pragma unroll 1
    for (; j < min(12, cols); ++j) column(Left<8>{}, j);
#pragma unroll 1
    for (; j < min(16, cols); ++j) column(Left<4>{}, j);
}
#endif

// The limbs' place in memory: 8 bytes, l first.
FIX64_FN int64_t pack(Limbs v) { return (int64_t)((uint64_t)(uint32_t)v.h << 32 | (uint32_t)v.l); }
FIX64_FN Limbs unpack(int64_t v) { return {(int32_t)v, (int32_t)(v >> 32)}; }

FIX64_FN int64_t join(Limbs v) {
    int64_t q = v.l;
    mad(q, v.h, int32_t(1) << 30);
    return q;
}

// Digits for the tensor cores: 4 q = sum of d_i 2^(8 (7 - i)), d_i in [-128, 127], kept as the bytes d_i + 128 of
// one 64-bit word (two bits more than q, so that the digits past the ones that are multiplied weigh less).
constexpr uint64_t kDigitBias = 0x8080808080808080ull;
FIX64_FN int64_t to_digits(int64_t q) { return (int64_t)(((uint64_t)q << 2) + kDigitBias); }
FIX64_FN int64_t from_digits(int64_t u) { return (int64_t)((uint64_t)u - kDigitBias) >> 2; }

// A cross sum starts here, so that total() rounds to nearest.
constexpr int64_t kCrossStart = int64_t(1) << 29;

// hh + cross in units of 2^-62.
FIX64_FN int64_t total(int64_t hh, int64_t cross) { return hh + (cross >> 30); }

// Moves the high part of the cross sum into hh.
FIX64_FN void fold(int64_t& hh, int64_t& cross) {
    hh += cross >> 30;
    cross &= (int64_t(1) << 30) - 1;
}

// Scale exponent of a row from its diagonal entry: a_ii * 4^-e in [1/16, 1/4). False for a diagonal
// that no positive definite matrix has (zero, negative, infinite, NaN).
FIX64_FN bool scale_exponent(double aii, int& e) {
    uint64_t const u = bits_of(aii);
    int const field = (int)(u >> 52);
    if (field >= 0x7ff || u == 0) {
        e = 0;
        return false;
    }
    e = ((field != 0 ? field - 1023 : -1011 - clz64(u)) + 4) >> 1;  // floor(log2 aii) + 4, halved
    return true;
}

// The threshold below which an entry is weak is 2^-(16 + weak_shift(n)): 2^-61 of error is 10 n 2^-52 of it, or less.
FIX64_FN int weak_shift(int n) { return (n >= 34) + (n >= 68) + (n >= 136) + (n >= 272); }
// The same in the high words of numbers in units of 2^-62.
FIX64_FN uint32_t weak_below(int n) { return (uint32_t(1) << 14) >> weak_shift(n); }
// Whether entry (i, j)'s remainder t = l_ij l_jj is below it.
FIX64_FN bool weak(int64_t t, uint32_t below) { return (uint32_t)hi32(t) + below < 2 * below; }
// The high word of the product of two entries with these high limbs.
FIX64_FN uint32_t term(int32_t h1, int32_t h2) {
    uint64_t const a = (uint32_t)(h1 < 0 ? -h1 : h1), b = (uint32_t)(h2 < 0 ? -h2 : h2);
    return (uint32_t)(a * b >> 32);
}

// Sum of squares of the high limbs of a row's entries in a panel: 16 of them fit 64 bits without a sign, and
// norm_of makes units of 2^-26 of them.
FIX64_FN void add_square(int64_t& sum, int32_t h) { mad(sum, h, h); }
FIX64_FN uint32_t norm_of(int64_t sum) { return (uint32_t)((uint64_t)sum >> 36); }
// 1/4, and more than what rounding the limbs may add.
constexpr uint32_t kNormMost = (uint32_t(1) << 24) + (uint32_t(1) << 10);
// A row's word: the sum of squares; whether its entries of the panel at hand are left to binary64; and its first
// panel with an entry other than zero before the diagonal, or a later one. A new row's word, and the word after panel
// J with these squares (any: there was such an entry).
constexpr uint32_t kNormMask = (uint32_t(1) << 26) - 1, kTodo = uint32_t(1) << 26, kNewRow = uint32_t(31) << 27;
FIX64_FN int first_panel(uint32_t word) { return (int)(word >> 27); }
FIX64_FN uint32_t row_after(uint32_t word, int J, int64_t squares, bool any) {
    uint32_t const norm = (word & kNormMask) + norm_of(squares), first = any && J < first_panel(word) ? (uint32_t)J : word >> 27;
    return (norm < kNormMask ? norm : kNormMask) | (word & kTodo) | first << 27;
}

// a * 2^-scale in units of 2^-62 (scale = e_i + e_j), truncated. False if |a| * 2^-scale is not below
// 1/4 (or a is not finite): the matrix is then not positive definite.
FIX64_FN bool from_double(double a, int scale, int64_t& out) {
    uint64_t const u = bits_of(a);
    int const field = (int)(u >> 52) & 0x7ff;
    uint64_t const m = (u & ((uint64_t(1) << 52) - 1)) | (uint64_t)(field != 0) << 52;
    int const r = scale + 1020 - (field != 0 ? field : 1);  // a = m * 2^7 * 2^(scale - 62 - r)
    int64_t const v = (int64_t)((m << 7) >> ((uint32_t)r < 63u ? r : 63));
    int64_t const sign = (int64_t)u >> 63;
    out = (v ^ sign) - sign;
    return r >= 0 || m == 0;
}

// q * 2^e for a factor entry: |q| <= 2^61 and a scale exponent's e, so that the result is normal or 0.
FIX64_FN double entry_to_double(int64_t q, int e) {
#ifdef __CUDA_ARCH__
    double const d = (double)q;
    return q == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + (e << 20), __double2loint(d));
#else
    return __builtin_ldexp((double)q, e);
#endif
}

// A pivot's reciprocal square root 1/sqrt(s * 2^-62) = r * 2^u, r in (1, 2], as two 31-bit limbs of
// r * 2^61. top = 2^(29 - u).
struct alignas(16) Rsqrt {
    int32_t l, h, u, top;
};

// The smallest pivot, 2^-42 to 2^-40 of its diagonal entry. Binary64's error of a pivot is at most about
// (n + 1) 2^-53 of the diagonal entry, 2^-44 for n = 512, so above this both find it positive.
constexpr int64_t kPivotMin = int64_t(1) << 18;

// s in [kPivotMin, 2^62). Halley's iteration (one term beyond Newton) on the hardware's binary32
// estimate: with e = 1 - v y^2, y (1 + e/2 + 3 e^2/8) has a relative error of 5/16 |e|^3, below
// 2^-62 for the estimate's |e| < 2^-20. The products keep the terms above 2^-60.
FIX64_FN Rsqrt pivot_rsqrt(int64_t s) {
    int const z = clz64((uint64_t)s) & ~1;       // s << z in [2^62, 2^64)
    uint64_t const v = (uint64_t)s << z;         // v * 2^-64 in [1/4, 1)
    int const u = (z >> 1) - 1;
    uint32_t const vh = (uint32_t)(v >> 32), vl = (uint32_t)v;
    uint32_t y = (uint32_t)(approx_rsqrt((float)vh) * 70368744177664.0f);  // 2^30 / sqrt(v), at most 2^31
    y = y > 0x7fffffffu ? 0x7fffffffu : y;
    uint64_t const yy = (uint64_t)y * y;
    uint32_t const ph = (uint32_t)(yy >> 32), pl = (uint32_t)yy;
    uint64_t const w = (uint64_t)vh * ph + umul_hi32(vh, pl) + umul_hi32(vl, ph);  // v y^2, units of 2^-60
    int64_t const e = (int64_t(1) << 60) - (int64_t)w;
    int32_t const t = (int32_t)(e >> 20);
    int64_t tt = 0;
    mad(tt, t, t);
    int64_t c8 = e << 2;  // 8 (e/2 + 3 e^2/8)
    mad(c8, (int32_t)(tt >> 20), 3);
    int64_t r = ((int64_t)y << 31) + umul_hi32(y, lo32(c8));  // y + y * c8 / 8, units of 2^-61
    mad(r, (int32_t)y, hi32(c8));
    bool const two = (r >> 62) != 0;
    return {two ? 0x7fffffff : (int32_t)(lo32(r) & 0x7fffffffu), two ? 0x7fffffff : (int32_t)(r >> 31), u,
            int32_t(1) << (29 - u)};
}

// t / sqrt(pivot): a remainder in units of 2^-62 becomes an entry in units of 2^-61, truncated. False if the
// entry reaches kEntryMost.
FIX64_FN bool scale_entry(int64_t t, Rsqrt y, int64_t& q) {
    bool const ok = (uint32_t)(hi32(t) + y.top) < 2u * (uint32_t)y.top;  // |t| <= 2^(61 - u)
    uint64_t const w = (uint64_t)t << (y.u & 31);
    int32_t const h = (int32_t)((int64_t)w >> 31), l = (int32_t)((uint32_t)w & 0x7fffffffu);
    int64_t cross = 0;
    mad(cross, h, y.l);
    mad(cross, l, y.h);
    q = cross >> 31;
    mad(q, h, y.h);
    constexpr uint32_t kMost = (uint32_t)(kEntryMost >> 32);
    return ok && (uint32_t)hi32(q) + kMost < 2 * kMost;
}

}  // namespace fix64
}  // namespace blastgpu
