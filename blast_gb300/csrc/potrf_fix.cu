// Batched binary64 Cholesky factorisation in 64-bit fixed point (fix64.cuh), 16 < n <= 512, sm_103a.
//
// Reference: blast::potrf (dense/Potrf.hpp:66-106): left-looking; a column strip takes the products
// of all earlier columns (the ger(-1, ...) loop), is factored on the diagonal and solved below it.
//
// What bounds it: in binary64 the multiply-adds, 2 lanes a clock and SM whatever the mapping (33.6 ms for
// 2,048 matrices with n uniform in 64 .. 512, factored and solved with one right-hand side). In fixed
// point the integer multiplications and additions, six instructions a product on two pipes (9.3 ms for
// the same batch), with the matrix's rows scaled; binary64 is left with one conversion per factor entry.
//
// Mapping: one CTA of T threads per matrix, panels of 16 columns, the rows of a panel in chunks of T.
//  * Update: each thread holds a 4 x 4 tile of the T x 16 chunk (rows T/4 apart, adjacent columns;
//    64 registers of sums), the earlier columns come through shared memory 16 at a time, double
//    buffered with cp.async. A step costs 48 multiply-adds against 4 row loads and 2 (16-byte)
//    column loads, all free of bank conflicts.
//  * The first chunk's first 32 rows: one warp, a row per lane, the 16 columns right-looking in
//    registers, the pivot row's limbs by shuffles. The reciprocal square root is integer as well.
//  * Other rows: a row per thread against the diagonal block, left-looking in registers.
//  * The factor stays in fixed point in the workspace (L itself, unless the caller says otherwise),
//    where the later panels read it, and becomes binary64 in one last pass.
//
// Panels of 16 keep the work inside a panel, which runs at a lower rate, at 8 n^2 of the n^3 / 6
// products, and let all T threads own a row of it.
#include "common.cuh"
#include "fix64.cuh"

namespace blastgpu {
namespace {

using fix64::Limbs;
using fix64::Rsqrt;

constexpr int kNB = 16;

template <int T>
struct Shape {
    static constexpr int NMAX = T == 32 ? 64 : T == 64 ? 128 : 512;  // largest n that runs with T threads
    static constexpr int RT = T / 4;    // distance of a thread's rows
    static constexpr int RS = T + kNB;  // staged column: the chunk's rows, then the diagonal block's
    static constexpr int CS = T + 2;    // column stride of the chunk: 4 columns x 8 rows hit all banks
    static constexpr int kStage = 0;
    static constexpr int kChunk = kStage + 2 * kNB * RS * 8;
    static constexpr int kDiag = kChunk + kNB * CS * 8;
    static constexpr int kRsqrt = kDiag + kNB * kNB * 8;
    static constexpr int kScale = kRsqrt + kNB * 16;
    static constexpr int kBad = kScale + NMAX * 4;
    static constexpr int kBytes = kBad + NMAX;
};

template <int T>
__device__ __forceinline__ void cta_sync() {
    if constexpr (T == 32) __syncwarp();
    else __syncthreads();
}

__device__ __forceinline__ void cp_async8(Limbs* dst, const Limbs* src) {
    unsigned const d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

// Columns 16 s .. 16 s + 15 of the workspace, rows k0 + r0 .. of the chunk; below the first chunk
// also the diagonal block's rows.
template <int T>
__device__ __forceinline__ void stage_columns(Limbs* stage, const Limbs* W, int64_t ldw, int k0, int r0, int mr, int nb,
                                              int s) {
    using S = Shape<T>;
    Limbs* dst = stage + (s & 1) * kNB * S::RS;
    Limbs const* src = W + k0 + (int64_t)(kNB * s) * ldw;
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

// The chunk's remainders A - L L^T over the columns before k0, into C (units of 2^-62). RA: rows per
// thread that the chunk needs. Rows past mr and columns past nb hold whatever shared memory held; they
// are not used.
template <int T, int RA>
__device__ __forceinline__ void update_chunk(int k0, int r0, int mr, int nb, const double* A, int64_t lda,
                                             const Limbs* W, int64_t ldw, Limbs* stage, int64_t* C, const int* scale,
                                             unsigned char* bad) {
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
        if (!ok && r < mr) bad[k0 + r0 + r] = fix64::kNoPivot | fix64::kOutOfRange;
    }
    Limbs const* colbase = stage + (r0 == 0 ? ct : T + ct);
    Limbs const* rowbase = stage + rt;
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
                Limbs const v = rowbase[base + q * S::RS + S::RT * i];
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

// The panel's first 32 rows (mr of them exist), one warp, a row per lane: the 16 columns right-looking.
// Leaves the diagonal block's entries in D, the pivots' reciprocal square roots in rsq, the entries
// in W. Returns the number of columns factored (nb unless a pivot is not positive).
template <int T>
__device__ __forceinline__ int factor_diagonal(int k0, int mr, int nb, const int64_t* C, Limbs* W, int64_t ldw, Limbs* D,
                                               Rsqrt* rsq, unsigned char* bad) {
    using S = Shape<T>;
    int const lane = threadIdx.x & 31;
    bool const mine = lane < mr;
    int64_t acc[kNB], cr[kNB];
#pragma unroll
    for (int c = 0; c < kNB; ++c) {
        acc[c] = mine && c < nb ? C[c * S::CS + lane] : 0;
        cr[c] = fix64::kCrossStart;
    }
    bool const no_pivot = mine && bad[k0 + lane] != 0;
    bool off = false;
    int done = nb;
#pragma unroll
    for (int j = 0; j < kNB; ++j) {
        if (j < done) {  // warp-uniform
            int64_t const t = acc[j] - fix64::total(0, cr[j]);
            int64_t const s = __shfl_sync(0xffffffffu, off || no_pivot ? (int64_t)-1 : t, j);
            if (s < fix64::kPivotMin) {
                done = j;
            } else {
                Rsqrt const y = fix64::pivot_rsqrt(s);
                int64_t q;
                bool const ok = fix64::scale_entry<fix64::kEntryBits>(t, y, q);
                off |= !ok && lane > j;
                Limbs const v = fix64::split(q);
                if (lane >= j && mine) W[(k0 + lane) + (int64_t)(k0 + j) * ldw] = v;
                if (lane < kNB) D[lane * kNB + j] = v;
                if (lane == 0) rsq[j] = y;
#pragma unroll
                for (int c = j + 1; c < kNB; ++c) {
                    int const h = __shfl_sync(0xffffffffu, v.h, c), l = __shfl_sync(0xffffffffu, v.l, c);
                    fix64::mad(acc[c], -v.h, h);
                    fix64::mad(cr[c], v.h, l);
                    fix64::mad(cr[c], v.l, h);
                }
            }
        }
    }
    if (off) bad[k0 + lane] = fix64::kNoPivot | fix64::kOutOfRange;
    return done;
}

// Row r of the chunk against the diagonal block (its first `done` columns), one thread.
template <int T>
__device__ __forceinline__ void solve_row(int row, int r, int k0, int done, const int64_t* C, Limbs* W, int64_t ldw,
                                          const Limbs* D, const Rsqrt* rsq, unsigned char* bad) {
    using S = Shape<T>;
    Limbs x[kNB];
    bool ok = true;
#pragma unroll
    for (int j = 0; j < kNB; ++j) {
        if (j < done) {
            int64_t hh = 0, c0 = fix64::kCrossStart, c1 = 0;
#pragma unroll
            for (int q = 0; q < j; ++q) {
                Limbs const d = D[j * kNB + q];
                fix64::mad(hh, x[q].h, d.h);
                fix64::mad(c0, x[q].h, d.l);
                fix64::mad(c1, x[q].l, d.h);
            }
            int64_t const t = C[j * S::CS + r] - fix64::total(hh, c0 + c1);
            int64_t v;
            ok &= fix64::scale_entry<fix64::kEntryBits>(t, rsq[j], v);
            x[j] = fix64::split(v);
            W[row + (int64_t)(k0 + j) * ldw] = x[j];
        }
    }
    if (!ok) bad[row] = fix64::kNoPivot | fix64::kOutOfRange;
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
__global__ void __launch_bounds__(T, 512 / T) potrf_fix_kernel(Batch batch, int32_t* info) {
    using S = Shape<T>;
    extern __shared__ __align__(16) unsigned char smem[];
    Limbs* stage = reinterpret_cast<Limbs*>(smem + S::kStage);
    int64_t* C = reinterpret_cast<int64_t*>(smem + S::kChunk);
    Limbs* D = reinterpret_cast<Limbs*>(smem + S::kDiag);
    Rsqrt* rsq = reinterpret_cast<Rsqrt*>(smem + S::kRsqrt);
    int* scale = reinterpret_cast<int*>(smem + S::kScale);
    unsigned char* bad = smem + S::kBad;
    __shared__ int s_done;
    int64_t const b = blockIdx.x;
    FixItem it;
    if (!batch.get(b, it) || it.n > S::NMAX) return;
    int const n = it.n, tid = threadIdx.x;
    Limbs* W = reinterpret_cast<Limbs*>(it.W);
    for (int i = tid; i < n; i += T) {
        int e;
        bad[i] = fix64::scale_exponent(it.A[i + (int64_t)i * it.lda], e) ? 0 : fix64::kNoPivot;
        scale[i] = e;
    }
    cta_sync<T>();
    for (int i = tid; i < n; i += T) {
        if (bad[i]) {
            int e = scale[i];
            for (int j = 0; j < i; ++j)
                if (!bad[j]) e = max(e, fix64::exponent_of(it.A[i + (int64_t)j * it.lda]) - scale[j] + fix64::kGrowth);
            scale[i] = e;
        }
    }
    cta_sync<T>();
    int good = n;  // columns factored
    for (int k0 = 0; k0 < n; k0 += kNB) {
        int const nb = min(kNB, n - k0), m = n - k0;
        int done = nb;
        for (int r0 = 0; r0 < m; r0 += T) {
            int const mr = min(T, m - r0);
#define BLASTGPU_UPDATE(RA) \
    update_chunk<T, RA>(k0, r0, mr, nb, it.A, it.lda, W, it.ldw, stage, C, scale, bad)
            switch ((mr + S::RT - 1) / S::RT) {
                case 1: BLASTGPU_UPDATE(1); break;
                case 2: BLASTGPU_UPDATE(2); break;
                case 3: BLASTGPU_UPDATE(3); break;
                default: BLASTGPU_UPDATE(4); break;
            }
#undef BLASTGPU_UPDATE
            cta_sync<T>();
            if (r0 == 0) {
                if (tid < 32) {
                    done = factor_diagonal<T>(k0, mr, nb, C, W, it.ldw, D, rsq, bad);
                    if (tid == 0) s_done = done;
                }
                cta_sync<T>();
                done = s_done;
            }
            if (tid < mr && (r0 > 0 || tid >= 32))
                solve_row<T>(k0 + r0 + tid, tid, k0, done, C, W, it.ldw, D, rsq, bad);
            cta_sync<T>();  // C is written again; the panel's columns are read from now on
        }
        if (done < nb) {
            good = k0 + done;
            break;
        }
    }
    if (info && tid == 0) info[b] = good < n ? good + 1 : 0;
    // Fixed point to binary64, a warp per column. After a pivot that is not positive the columns from it
    // on are NaN, and so are the rows whose entries left the fixed-point range.
    double const nan = __longlong_as_double(0x7ff8000000000000ll);
    int const lane = tid & 31, warp = tid >> 5;
    for (int c = warp; c < n; c += T / 32) {
        Limbs const* w = W + (int64_t)c * it.ldw;
        double* l = it.L + (int64_t)c * it.ldl;
        for (int i0 = c; i0 < n; i0 += 128) {
            Limbs v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                int const i = i0 + lane + 32 * u;
                v[u] = i < n && c < good ? w[i] : Limbs{0, 0};
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                int const i = i0 + lane + 32 * u;
                if (i < n) {
                    double x = fix64::entry_to_double(fix64::join(v[u]), scale[i] - 61);
                    if (c >= good || (bad[i] & fix64::kOutOfRange)) x = nan;
                    l[i] = x;
                    if (it.L2) it.L2[i + (int64_t)c * it.ldl2] = x;
                }
            }
        }
    }
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
