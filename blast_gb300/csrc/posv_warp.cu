// Ragged Cholesky solves for small n (n <= 128), binary64: one warp per matrix. Matrices of kFixMinN
// rows and more arrive factored (potrf_fix.cu); smaller ones are factored here.
//
// Reference: blast::potrf (dense/Potrf.hpp:66-106), left-looking in strips of 4 columns: each
// element of a strip first takes the fused products of all earlier columns in ascending order
// (the ger(-1, ...) loop), then RegisterMatrix::potrf / ::trsm (RegisterMatrix.hpp:566-602,
// 710-739) finish the strip column by column. The solves follow dense/Trsm.hpp:39-65.
//
// Mapping: lane l owns rows l, l + 32, ... of its matrix (MAXT row blocks). Every element sees the
// same fused multiply-adds, in the same order, as the thread-per-matrix kernel, so the factor and
// the solutions are the same bits. A thread per matrix needs far more matrices than a ragged batch
// of small n has to fill the chip, and a CTA per matrix spends its time on barriers; a warp per
// matrix has neither problem.
//
// Solves, one right-hand side at a time: the forward substitution is a column sweep (once x_l is
// final, every row below takes its term), which keeps each row's ascending order. The backward
// substitution keeps the thread-per-matrix kernel's order for row i of the 4-row block i0 .. i0+3:
// first the rows below the block in ascending order, then the block's own later rows. That leaves four
// chains per matrix, and an instruction on the binary64 pipe takes its 64 cycles for 4 lanes as for 32,
// so one warp runs the backward substitution of the CTA's eight matrices, four lanes each. 4,096
// matrices of 32..128 rows, solved and differentiated: 2.18 ms with all their kernels, 2.67 ms with a warp
// to each matrix in both directions.
#include "common.cuh"

namespace blastgpu {
namespace {

constexpr int kWarpsPerCta = 8;  // an instance each; four lanes of one warp each in the backward substitution

struct Factor {
    const double* L;
    int64_t ld;
    int n;
};

// Column C of the strip at k of a matrix with at most 32 rows, lane = row: the terms of the strip's columns
// j < C (their final, scaled values), then the scaling by y = rsqrt_nr(pivot).
template <int C>
__device__ __forceinline__ void strip_column(double (&acc)[4], int k, int n, int lane, int& info) {
    int const owner = k + C;
    bool const mine = lane - k >= C && lane < n;
#pragma unroll
    for (int j = 0; j < C; ++j) {
        // l_{k+C, k+j}: row k + C's final value in column j, from the lane that holds it
        double const lcj = __shfl_sync(0xffffffffu, acc[j], owner);
        if (mine) acc[C] = fma(-lcj, acc[j], acc[C]);
    }
    double const s = __shfl_sync(0xffffffffu, acc[C], owner);
    if (!(s > 0.0) && info == 0) info = k + C + 1;
    double const y = rsqrt_nr(s);
    if (mine) acc[C] *= y;
}

// Left-looking Cholesky of the n x n matrix A (lower triangle read) into L (lower triangle
// written), n < kFixMinN, one warp. Returns 0 or the first bad pivot + 1, the same in every lane.
__device__ int warp_potrf(int n, const double* A, int lda, double* L, int ldl, int lane) {
    int info = 0;
    for (int k = 0; k < n; k += 4) {
        int const nc = min(4, n - k);
        bool const below = lane < n && lane >= k;
        double acc[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[c] = (c < nc && lane < n && lane - k >= c) ? A[lane + (int64_t)(k + c) * lda] : 0.0;
        // the earlier columns in ascending order
        for (int l = 0; l < k; ++l) {
            double const* col = L + (int64_t)l * ldl;
            double const a = below ? col[lane] : 0.0;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                double const b = c < nc ? col[k + c] : 0.0;
                if (lane - k >= c) acc[c] = fma(-a, b, acc[c]);
            }
        }
        strip_column<0>(acc, k, n, lane, info);
        if (nc > 1) strip_column<1>(acc, k, n, lane, info);
        if (nc > 2) strip_column<2>(acc, k, n, lane, info);
        if (nc > 3) strip_column<3>(acc, k, n, lane, info);
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (c < nc && lane < n && lane - k >= c) L[lane + (int64_t)(k + c) * ldl] = acc[c];
        __syncwarp();  // the strip's columns are read by every lane from the next strip on
    }
    return info;
}

// Columns l of the forward sweep with l in block TL (32 TL <= l < 32 TL + 32): rows in blocks
// below TL all take the term; block TL only below l.
template <int MAXT, int TL>
__device__ __forceinline__ void fwd_sweep_block(int n, const double* L, int ldl, double (&acc)[MAXT],
                                                double const (&d)[MAXT], int lane) {
    int const l1 = min(n, 32 * TL + 32);
    for (int l = 32 * TL; l < l1; ++l) {
        double col[MAXT];
        double const* cl = L + (int64_t)l * ldl;
#pragma unroll
        for (int t = TL; t < MAXT; ++t) {
            int const i = lane + 32 * t;
            col[t] = (i > l && i < n) ? cl[i] : 0.0;
        }
        double const xl = __shfl_sync(0xffffffffu, acc[TL] * d[TL], l & 31);
#pragma unroll
        for (int t = TL; t < MAXT; ++t) {
            int const i = lane + 32 * t;
            if (i == l) acc[t] = xl;
            else if (i > l && i < n) acc[t] = fma(-col[t], xl, acc[t]);
        }
    }
}

// y = L^{-1} b, one warp, column sweep; xs, rd: y and the reciprocals of L's diagonal (shared memory).
template <int MAXT>
__device__ __forceinline__ void warp_forward(int n, const double* L, int ldl, const double* bcol, double* xs,
                                             double* rd, int lane) {
    double acc[MAXT], d[MAXT];
#pragma unroll
    for (int t = 0; t < MAXT; ++t) {
        int const i = lane + 32 * t;
        acc[t] = i < n ? bcol[i] : 0.0;
        d[t] = i < n ? rcp_nr(L[i + (int64_t)i * ldl]) : 0.0;
    }
    fwd_sweep_block<MAXT, 0>(n, L, ldl, acc, d, lane);
    if constexpr (MAXT > 1) fwd_sweep_block<MAXT, (MAXT > 1 ? 1 : 0)>(n, L, ldl, acc, d, lane);
    if constexpr (MAXT > 2) fwd_sweep_block<MAXT, (MAXT > 2 ? 2 : 0)>(n, L, ldl, acc, d, lane);
    if constexpr (MAXT > 3) fwd_sweep_block<MAXT, (MAXT > 3 ? 3 : 0)>(n, L, ldl, acc, d, lane);
#pragma unroll
    for (int t = 0; t < MAXT; ++t) {
        int const i = lane + 32 * t;
        if (i < n) {
            xs[i] = acc[t];
            rd[i] = d[t];
        }
    }
}

// The same for n <= 32 MAXT rows: the number of row blocks fixes the register tiles, so the blocks past
// the last row cost nothing.
template <int MAXT>
__device__ __forceinline__ void forward_rows(int n, const double* L, int ldl, const double* bcol, double* xs,
                                             double* rd, int lane) {
    switch ((n + 31) >> 5) {
        case 0: break;
        case 1: warp_forward<1>(n, L, ldl, bcol, xs, rd, lane); break;
        case 2: if constexpr (MAXT >= 2) warp_forward<(MAXT >= 2 ? 2 : 1)>(n, L, ldl, bcol, xs, rd, lane); break;
        case 3: if constexpr (MAXT >= 3) warp_forward<(MAXT >= 3 ? 3 : 1)>(n, L, ldl, bcol, xs, rd, lane); break;
        default: if constexpr (MAXT >= 4) warp_forward<(MAXT >= 4 ? 4 : 1)>(n, L, ldl, bcol, xs, rd, lane); break;
    }
}

// Rows l .. l+7 of a column of L, zero from row n on: a term of two zeros leaves its sum as it is.
__device__ __forceinline__ void column_rows(double (&v)[8], const double* col, int l, int n) {
#pragma unroll
    for (int u = 0; u < 8; ++u) v[u] = l + u < n ? col[l + u] : 0.0;
}

// x = L^{-T} y of the CTA's instances by one warp, four lanes per instance (n = 0: none), in 4-row blocks
// from the bottom: lane r of the four has row i0 + r. xs: y in, x out; rd: 1 / diag(L).
__device__ __forceinline__ void warp_backward(int n, const double* L, int64_t ldl, double* xs, const double* rd,
                                              int lane) {
    int const r = lane & 3;
    int i0 = ((n + 3) & ~3) - 4;
    int const steps = __reduce_max_sync(0xffffffffu, (unsigned)(n + 3) >> 2);
    double v[8], t[4];  // the next rows of the lane's column; its rows i0 .. i0+3
    auto block = [&](int k0) {
        int const i = k0 + r;
        bool const on = k0 >= 0 && i < n;
        double const* col = L + (int64_t)(on ? i : 0) * ldl;
        column_rows(v, col, k0 + 4, on ? n : 0);
#pragma unroll
        for (int q = 1; q < 4; ++q) t[q] = on && q > r && k0 + q < n ? col[k0 + q] : 0.0;
    };
    block(i0);
    for (int step = 0; step < steps; ++step, i0 -= 4) {
        int const i = i0 + r;
        bool const on = i0 >= 0 && i < n;
        double s = on ? xs[i] : 0.0, tb[4];
        double const y = on ? rd[i] : 0.0;
        double const* col = L + (int64_t)(on ? i : 0) * ldl;
#pragma unroll
        for (int q = 1; q < 4; ++q) tb[q] = t[q];
        if (i0 >= 0) {
            int l = i0 + 4;
            for (; l + 8 < n; l += 8) {  // rows l .. l+7 while the next eight are on their way
                double w[8];
                column_rows(w, col, l + 8, on ? n : 0);
#pragma unroll
                for (int u = 0; u < 8; ++u) s = fma(-v[u], xs[l + u], s);
#pragma unroll
                for (int u = 0; u < 8; ++u) v[u] = w[u];
            }
            double w[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) w[u] = v[u];
            block(i0 - 4);
#pragma unroll
            for (int u = 0; u < 8; ++u) s = fma(-w[u], l + u < n ? xs[l + u] : 0.0, s);
        }
        __syncwarp();
        double xb[4];  // the block's own rows, each after its later rows in ascending order
#pragma unroll
        for (int p = 3; p >= 0; --p) {
            double e = s;
#pragma unroll
            for (int q = p + 1; q < 4; ++q) e = fma(-tb[q], xb[q], e);
            xb[p] = __shfl_sync(0xffffffffu, on ? e * y : 0.0, (lane & ~3) + p);
        }
        if (on) xs[i] = r == 0 ? xb[0] : r == 1 ? xb[1] : r == 2 ? xb[2] : xb[3];
        __syncwarp();
    }
}

// The CTA's substitutions for column c: one warp per instance forwards, all instances in warp 0 backwards.
// Called by all threads; n = 0: no instance, or none left. The solution stays in xs, complete for its own warp.
template <int MAXT>
__device__ __forceinline__ void cta_solve(int n, const double* L, int ldl, const double* bcol,
                                          double (&xs)[kWarpsPerCta][32 * MAXT], double (&rd)[kWarpsPerCta][32 * MAXT],
                                          Factor (&who)[kWarpsPerCta], int w, int lane) {
    forward_rows<MAXT>(n, L, ldl, bcol, xs[w], rd[w], lane);
    if (lane == 0) who[w] = Factor{L, ldl, n};
    __syncthreads();
    if (w == 0) {
        int const g = lane >> 2;
        Factor const f = who[g];
        warp_backward(f.n, f.L, f.ld, xs[g], rd[g], lane);
    }
    __syncthreads();
}

template <int MAXT>
__global__ void __launch_bounds__(kWarpsPerCta * 32) posv_warp_kernel(const blastgpu_posv_desc* desc, int64_t count,
                                                                     bool paired, int32_t* info) {
    __shared__ double xs[kWarpsPerCta][32 * MAXT], rd[kWarpsPerCta][32 * MAXT];
    __shared__ Factor who[kWarpsPerCta];
    int const w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int64_t const b = (int64_t)blockIdx.x * kWarpsPerCta + w;
    blastgpu_posv_desc const& dsc = desc[min(b, count - 1)];
    int const n = dsc.A.rows;
    // the launch's max_n bounds every instance; posv_pair.cu has solved the others
    bool const mine = b < count && n <= 32 * MAXT && !(paired && n >= kFixMinN && dsc.A.data != nullptr);
    if (mine && dsc.A.data != nullptr && n < kFixMinN) {  // else the factor is in L
        int const r = warp_potrf(n, dsc.A.data, dsc.A.ld, dsc.L.data, dsc.L.ld, lane);
        if (info && lane == 0) info[b] = r;
    }
    int const cols = mine && n > 0 ? dsc.B.cols : 0;
    for (int c = 0; __syncthreads_or(c < cols); ++c) {
        bool const on = c < cols;
        cta_solve<MAXT>(on ? n : 0, dsc.L.data, dsc.L.ld, on ? dsc.B.data + (int64_t)c * dsc.B.ld : nullptr, xs, rd,
                        who, w, lane);
        if (on)
            for (int i = lane; i < n; i += 32) dsc.X.data[i + (int64_t)c * dsc.X.ld] = xs[w][i];
        __syncwarp();
    }
}

// dl/dA = -(g x^T + x g^T)/2 of one instance with one right-hand side, g = dl/dB in xs: lanes over rows, a
// column at a time.
template <int NB>
__device__ __forceinline__ void warp_outer(blastgpu_posv_bwd_desc const& d, int n, const double* xs, int lane) {
    double xi[NB], gi[NB];
#pragma unroll
    for (int t = 0; t < NB; ++t) {
        int const i = lane + 32 * t;
        xi[t] = i < n ? d.X.data[i] : 0.0;
        gi[t] = i < n ? xs[i] : 0.0;
    }
    for (int j = 0; j < n; ++j) {
        double const xj = d.X.data[j], gj = xs[j];
        double* ga = d.Abar.data + (int64_t)j * d.Abar.ld;
#pragma unroll
        for (int t = 0; t < NB; ++t) {
            int const i = lane + 32 * t;
            if (i < n) ga[i] = -0.5 * fma(xi[t], gj, gi[t] * xj);
        }
    }
}

// Adjoint of X = A^{-1} B, one warp per instance (as posv_bwd_kernel, which runs a CTA per matrix): the
// factor kept in L or recomputed from A, dl/dB = A^{-1} dl/dX with the same solve, then
// dl/dA = -(dl/dB X^T + X dl/dB^T)/2.
template <int MAXT>
__global__ void __launch_bounds__(kWarpsPerCta * 32) posv_bwd_warp_kernel(const blastgpu_posv_bwd_desc* desc,
                                                                         int64_t count, int recompute, int32_t* info) {
    __shared__ double xs[kWarpsPerCta][32 * MAXT], rd[kWarpsPerCta][32 * MAXT];
    __shared__ Factor who[kWarpsPerCta];
    int const w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int64_t const b = (int64_t)blockIdx.x * kWarpsPerCta + w;
    blastgpu_posv_bwd_desc const& d = desc[min(b, count - 1)];
    int const n = d.A.rows;
    bool const mine = b < count && n <= 32 * MAXT;  // the launch's max_n bounds every instance
    if (mine && recompute && n < kFixMinN) {        // else the factor is in L
        int const r = warp_potrf(n, d.A.data, d.A.ld, d.L.data, d.L.ld, lane);
        if (info && lane == 0) info[b] = r;
    } else if (mine && !recompute && info && lane == 0) {
        info[b] = 0;
    }
    int const nrhs = mine && n > 0 ? d.X.cols : 0;
    for (int c = 0; __syncthreads_or(c < nrhs); ++c) {
        bool const on = c < nrhs;
        cta_solve<MAXT>(on ? n : 0, d.L.data, d.L.ld, on ? d.Xbar.data + (int64_t)c * d.Xbar.ld : nullptr, xs, rd, who,
                        w, lane);
        if (on)
            for (int i = lane; i < n; i += 32) d.Bbar.data[i + (int64_t)c * d.Bbar.ld] = xs[w][i];
        __syncwarp();
    }
    if (!mine || n == 0) return;
    if (nrhs == 1) {  // dl/dB is still in xs
        switch ((n + 31) >> 5) {
            case 1: warp_outer<1>(d, n, xs[w], lane); break;
            case 2: if constexpr (MAXT >= 2) warp_outer<(MAXT >= 2 ? 2 : 1)>(d, n, xs[w], lane); break;
            case 3: if constexpr (MAXT >= 3) warp_outer<(MAXT >= 3 ? 3 : 1)>(d, n, xs[w], lane); break;
            default: if constexpr (MAXT >= 4) warp_outer<(MAXT >= 4 ? 4 : 1)>(d, n, xs[w], lane); break;
        }
        return;
    }
    for (int j = 0; j < n; ++j)
        for (int i = lane; i < n; i += 32) {
            double acc = 0.0;
            for (int c = 0; c < nrhs; ++c) {
                acc = fma(d.Bbar.data[i + (int64_t)c * d.Bbar.ld], d.X.data[j + (int64_t)c * d.X.ld], acc);
                acc = fma(d.X.data[i + (int64_t)c * d.X.ld], d.Bbar.data[j + (int64_t)c * d.Bbar.ld], acc);
            }
            d.Abar.data[i + (int64_t)j * d.Abar.ld] = -0.5 * acc;
        }
}

}  // namespace

// Adjoints of ragged binary64 Cholesky solves with every n <= 128, one warp per matrix
// (blastgpu_dposv_bwd_batched routes such launches here unless "posv.warp_bwd.n<bin>" is 0).
int launch_posv_bwd_warp(const blastgpu_posv_bwd_desc* desc, int64_t count, int max_n, int recompute, int32_t* info,
                         cudaStream_t s) {
    if (count == 0) return BLASTGPU_SUCCESS;
    int64_t const blocks = (count + kWarpsPerCta - 1) / kWarpsPerCta;
    if (blocks > 0x7fffffff) return BLASTGPU_ERR_TOO_LARGE;
    if (recompute && max_n >= kFixMinN) {
        int const st = launch_potrf_fix(desc, kFixMinN, max_n, info, count, s);
        if (st != BLASTGPU_SUCCESS) return st;
    }
    unsigned const g = (unsigned)blocks, t = kWarpsPerCta * 32;
    if (max_n <= 32) posv_bwd_warp_kernel<1><<<g, t, 0, s>>>(desc, count, recompute, info);
    else if (max_n <= 64) posv_bwd_warp_kernel<2><<<g, t, 0, s>>>(desc, count, recompute, info);
    else if (max_n <= 128) posv_bwd_warp_kernel<4><<<g, t, 0, s>>>(desc, count, recompute, info);
    else return BLASTGPU_ERR_TOO_LARGE;
    return check_launch();
}

// Ragged binary64 Cholesky solves with every n <= 128, one warp per matrix (blastgpu_dposv_batched
// routes such launches here unless "posv.warp.n<bin>" is 0).
int launch_posv_warp(const blastgpu_posv_desc* desc, int64_t count, int max_n, int32_t* info, cudaStream_t s) {
    if (count == 0) return BLASTGPU_SUCCESS;
    int64_t const blocks = (count + kWarpsPerCta - 1) / kWarpsPerCta;
    if (blocks > 0x7fffffff) return BLASTGPU_ERR_TOO_LARGE;
    bool const paired = max_n <= kPairMaxN;
    if (max_n >= kFixMinN) {
        int const st = paired ? launch_posv_pair(desc, kFixMinN, max_n, info, count, s)
                              : launch_potrf_fix(desc, kFixMinN, max_n, info, count, s);
        if (st != BLASTGPU_SUCCESS) return st;
    }
    unsigned const g = (unsigned)blocks, t = kWarpsPerCta * 32;
    if (max_n <= 32) posv_warp_kernel<1><<<g, t, 0, s>>>(desc, count, paired, info);
    else if (max_n <= 64) posv_warp_kernel<2><<<g, t, 0, s>>>(desc, count, paired, info);
    else if (max_n <= 128) posv_warp_kernel<4><<<g, t, 0, s>>>(desc, count, paired, info);
    else return BLASTGPU_ERR_TOO_LARGE;
    return check_launch();
}

}  // namespace blastgpu
