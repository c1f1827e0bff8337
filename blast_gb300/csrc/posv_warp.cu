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
// first the rows below the block in ascending order, then the block's own later rows. It runs
// one block at a time from the bottom: four lanes take the rows below, then lane 0 finishes the
// block.
#include "common.cuh"

namespace blastgpu {
namespace {

constexpr int kWarpsPerCta = 4;

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

// X(:, j) = A^{-1} B(:, j) from the factor L, one warp; xs: n doubles of shared memory.
template <int MAXT>
__device__ void warp_potrs_column(int n, const double* L, int ldl, const double* bcol, double* xcol, double* xs,
                                  int lane) {
    // forward: L y = b, column sweep
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
        if (i < n) xs[i] = acc[t];
    }
    __syncwarp();
    // backward: L^T x = y, 4-row blocks from the bottom
    __shared__ double part[kWarpsPerCta][4];
    int const w = threadIdx.x >> 5;
    for (int i0 = ((n - 1) / 4) * 4; i0 >= 0; i0 -= 4) {
        int const ni = min(4, n - i0);
        if (lane < ni) {
            int const i = i0 + lane;
            double const* li = L + (int64_t)i * ldl;  // column i of L: L(l, i) for l > i
            double s = xs[i];
            int l = i0 + 4;
            for (; l + 8 <= n; l += 8) {
                double v[8], x[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    v[u] = li[l + u];
                    x[u] = xs[l + u];
                }
#pragma unroll
                for (int u = 0; u < 8; ++u) s = fma(-v[u], x[u], s);
            }
            for (; l < n; ++l) s = fma(-li[l], xs[l], s);
            part[w][lane] = s;
        }
        __syncwarp();
        if (lane == 0) {
            double xb[4];
            for (int r = ni - 1; r >= 0; --r) {
                int const i = i0 + r;
                double s = part[w][r];
                for (int q = r + 1; q < ni; ++q) s = fma(-L[(i0 + q) + (int64_t)i * ldl], xb[q], s);
                xb[r] = s * rcp_nr(L[i + (int64_t)i * ldl]);
                xs[i] = xb[r];
            }
        }
        __syncwarp();
    }
    for (int i = lane; i < n; i += 32) xcol[i] = xs[i];
    __syncwarp();
}

// One instance with n <= 32 NB: its row blocks (NB of them) fix the register tiles, so the
// blocks past its last row cost nothing.
template <int NB>
__device__ __forceinline__ void warp_posv(blastgpu_posv_desc const& dsc, int n, double* xs, int lane, int32_t* info_b) {
    if (NB == 1 && dsc.A.data != nullptr && n < kFixMinN) {  // else the factor is in L
        int const r = warp_potrf(n, dsc.A.data, dsc.A.ld, dsc.L.data, dsc.L.ld, lane);
        if (info_b && lane == 0) *info_b = r;
    }
    for (int j = 0; j < dsc.B.cols; ++j)
        warp_potrs_column<NB>(n, dsc.L.data, dsc.L.ld, dsc.B.data + (int64_t)j * dsc.B.ld,
                              dsc.X.data + (int64_t)j * dsc.X.ld, xs, lane);
}

template <int MAXT>
__global__ void __launch_bounds__(kWarpsPerCta * 32) posv_warp_kernel(const blastgpu_posv_desc* desc, int64_t count,
                                                                     bool paired, int32_t* info) {
    __shared__ double xs_all[kWarpsPerCta][32 * MAXT];
    int const w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int64_t const b = (int64_t)blockIdx.x * kWarpsPerCta + w;
    if (b >= count) return;
    blastgpu_posv_desc const& dsc = desc[b];
    int const n = dsc.A.rows;
    if (n > 32 * MAXT) return;  // the launch's max_n bounds every instance
    if (paired && n >= kFixMinN && dsc.A.data != nullptr) return;  // solved by posv_pair.cu
    int32_t* const info_b = info ? info + b : nullptr;
    switch ((n + 31) >> 5) {
        case 0:
        case 1: warp_posv<1>(dsc, n, xs_all[w], lane, info_b); break;
        case 2: if constexpr (MAXT >= 2) warp_posv<(MAXT >= 2 ? 2 : 1)>(dsc, n, xs_all[w], lane, info_b); break;
        case 3: if constexpr (MAXT >= 3) warp_posv<(MAXT >= 3 ? 3 : 1)>(dsc, n, xs_all[w], lane, info_b); break;
        default: if constexpr (MAXT >= 4) warp_posv<(MAXT >= 4 ? 4 : 1)>(dsc, n, xs_all[w], lane, info_b); break;
    }
}

// Adjoint of X = A^{-1} B for one instance, one warp (as posv_bwd_kernel, which runs a CTA per
// matrix): the factor kept in L or recomputed from A, dl/dB = A^{-1} dl/dX with the warp's solve,
// dl/dA = -(dl/dB X^T + X dl/dB^T)/2 written by lanes over rows, a column at a time.
template <int NB>
__device__ __forceinline__ void warp_posv_bwd(blastgpu_posv_bwd_desc const& d, int n, int recompute, double* xs,
                                              int lane, int32_t* info_b) {
    if (NB == 1 && recompute && n < kFixMinN) {  // else the factor is in L
        int const r = warp_potrf(n, d.A.data, d.A.ld, d.L.data, d.L.ld, lane);
        if (info_b && lane == 0) *info_b = r;
    } else if (!recompute && info_b && lane == 0) {
        *info_b = 0;
    }
    int const nrhs = d.X.cols;
    for (int c = 0; c < nrhs; ++c)
        warp_potrs_column<NB>(n, d.L.data, d.L.ld, d.Xbar.data + (int64_t)c * d.Xbar.ld,
                              d.Bbar.data + (int64_t)c * d.Bbar.ld, xs, lane);
    if (nrhs == 1) {  // dl/dB is still in xs
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
        return;
    }
    __syncwarp();  // dl/dB columns are complete in memory
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

template <int MAXT>
__global__ void __launch_bounds__(kWarpsPerCta * 32) posv_bwd_warp_kernel(const blastgpu_posv_bwd_desc* desc,
                                                                         int64_t count, int recompute, int32_t* info) {
    __shared__ double xs_all[kWarpsPerCta][32 * MAXT];
    int const w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int64_t const b = (int64_t)blockIdx.x * kWarpsPerCta + w;
    if (b >= count) return;
    blastgpu_posv_bwd_desc const& d = desc[b];
    int const n = d.A.rows;
    if (n > 32 * MAXT) return;  // the launch's max_n bounds every instance
    int32_t* const info_b = info ? info + b : nullptr;
    switch ((n + 31) >> 5) {
        case 0:
        case 1: warp_posv_bwd<1>(d, n, recompute, xs_all[w], lane, info_b); break;
        case 2: if constexpr (MAXT >= 2) warp_posv_bwd<(MAXT >= 2 ? 2 : 1)>(d, n, recompute, xs_all[w], lane, info_b); break;
        case 3: if constexpr (MAXT >= 3) warp_posv_bwd<(MAXT >= 3 ? 3 : 1)>(d, n, recompute, xs_all[w], lane, info_b); break;
        default: if constexpr (MAXT >= 4) warp_posv_bwd<(MAXT >= 4 ? 4 : 1)>(d, n, recompute, xs_all[w], lane, info_b); break;
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
