// Batched gemm D = alpha*A*B + beta*C, binary64, sm_103a.
//
// Reference: blast::gemm (algorithm/Gemm.hpp:41-118) tiles D with register matrices
// (algorithm/arch/avx2/Tile.hpp:45-139) and runs, per tile, the rank-1 loop of
// register_matrix/Gemm.hpp:64-124:  acc = 0; for k: acc += a_k * b_k^T (fused); acc *= alpha;
// acc = fma(beta, C, acc); store.
//
// GPU mapping: one warp per instance. The warp's 32 lanes form a 4 x 8 grid; each lane owns an
// RM x RN register tile (BLAST's RegisterMatrix), so a warp tile is (4*RM) x (8*RN) (24 x 24 for
// RM = 6, RN = 3: every lane holds 18 accumulators and no lane idles). Operand panels of K_CHUNK
// columns of A and rows of B are staged in shared memory with coalesced loads; every lane then
// performs the same per-element sequence of fused multiply-adds as BLAST (ascending k, alpha
// scaling, fma(beta, c, .)), so the results are bit-identical to the oracle restatement.
// GB300's binary64 pipe (~1.2 TFLOP/s measured) bounds this kernel; the staging and shared-memory
// traffic are far below their own limits.
#include <cstdio>

#include "common.cuh"

namespace blastgpu {
namespace {

constexpr int kWarps = 4;    // warps (instances) per CTA
// K columns staged per pass: static shared memory stays under 48 KB, and the loads in flight within the
// registers of the CTAs below (32 columns took 508 instead of 359 us for 3,000 products of 57 x 39 x 23).
constexpr int kKChunk = 16;
// CTAs per SM that a tile's registers are bounded for.
template <int RM, int RN>
constexpr int kCtas = RM * RN <= 2 ? 9 : RM * RN <= 4 ? 7 : RM * RN <= 8 ? 6 : 4;

struct StridedGemm {
    int m, n, k;
    double alpha, beta;
    MatView A, B, C, D;
    int64_t sa, sb, sc, sd;
    __device__ void get(int64_t b, int& mm, int& nn, int& kk, double& al, double& be, MatView& a,
                        MatView& bm, MatView& c, MatView& d) const {
        mm = m; nn = n; kk = k; al = alpha; be = beta;
        a = A; a.p += b * sa;
        bm = B; bm.p += b * sb;
        c = C; c.p += b * sc;
        d = D; d.p += b * sd;
    }
};

struct DescGemm {
    const blastgpu_gemm_desc* desc;
    __device__ void get(int64_t b, int& mm, int& nn, int& kk, double& al, double& be, MatView& a,
                        MatView& bm, MatView& c, MatView& d) const {
        blastgpu_gemm_desc const& g = desc[b];
        mm = g.D.rows; nn = g.D.cols; kk = g.A.cols; al = g.alpha; be = g.beta;
        a = view(g.A); bm = view(g.B); c = view(g.C); d = view(g.D);
    }
};

// Adjoint of D = alpha*A*B + beta*C over descriptors (A, B as views, so op() is the view):
// which = 0 forms Abar += alpha*Dbar*B^T in A's orientation, which = 1 forms Bbar += alpha*A^T*Dbar
// in B's; both are gemms with beta = 1 on transposed views, in place. An instance whose shapes
// do not fit (gemm_bwd_ok) or whose gradient is not wanted (null data) gets m = 0.
__device__ __forceinline__ bool gemm_bwd_ok(blastgpu_gemm_bwd_desc const& g) {
    int const m = g.Dbar.rows, n = g.Dbar.cols, k = g.A.cols;
    blastgpu_mat t;
    if (!view_ok(g.Dbar) || g.A.rows != m || g.B.rows != k || g.B.cols != n) return false;
    if (g.Abar.data && !(view_ok(g.B) && transposed(g.B, t) && view_ok(g.Abar) && g.Abar.rows == m && g.Abar.cols == k))
        return false;
    if (g.Bbar.data && !(view_ok(g.A) && transposed(g.A, t) && view_ok(g.Bbar) && g.Bbar.rows == k && g.Bbar.cols == n))
        return false;
    if (g.Cbar.data && !(view_ok(g.Cbar) && g.Cbar.rows == m && g.Cbar.cols == n)) return false;
    return true;
}

struct GemmBwdBatch {
    const blastgpu_gemm_bwd_desc* desc;
    int which;
    __device__ void get(int64_t b, int& mm, int& nn, int& kk, double& al, double& be, MatView& a, MatView& bm,
                        MatView& c, MatView& d) const {
        blastgpu_gemm_bwd_desc const& g = desc[b];
        mm = nn = kk = 0;
        al = g.alpha;
        be = 1.0;
        if (!gemm_bwd_ok(g)) return;
        blastgpu_mat t;
        if (which == 0) {
            if (!g.Abar.data) return;
            transposed(g.B, t);
            mm = g.Abar.rows; nn = g.Abar.cols; kk = g.Dbar.cols;
            a = view(g.Dbar); bm = view(t); c = view(g.Abar);
        } else {
            if (!g.Bbar.data) return;
            transposed(g.A, t);
            mm = g.Bbar.rows; nn = g.Bbar.cols; kk = g.Dbar.rows;
            a = view(t); bm = view(g.Dbar); c = view(g.Bbar);
        }
        d = c;
    }
};

// Cbar += beta*Dbar (fma(beta, dbar, cbar), as the strided adjoint) and the status of every instance.
__global__ void __launch_bounds__(128) gemm_bwd_c_kernel(const blastgpu_gemm_bwd_desc* desc, int64_t count,
                                                         int32_t* status) {
    int64_t const b = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
    int const lane = threadIdx.x & 31;
    if (b >= count) return;
    blastgpu_gemm_bwd_desc const& g = desc[b];
    bool const ok = gemm_bwd_ok(g);
    if (status && lane == 0) status[b] = ok ? 0 : -1;
    if (!ok || !g.Cbar.data) return;
    MatView const Db = view(g.Dbar), Cb = view(g.Cbar);
    int const m = g.Dbar.rows, n = g.Dbar.cols;
    for (int e = lane; e < m * n; e += 32) {
        int const i = e % m, j = e / m;
        Cb(i, j) = fma(g.beta, Db(i, j), Cb(i, j));
    }
}

// Stages the W x KC panel of an operand whose element (r, q) (r along the tile, q along k) is V(r0 + r,
// q0 + q), or V(q0 + q, r0 + r) with SWAP, into dst[q][r]; zeros past `rows`. Lanes take consecutive elements
// of the storage. Elements with q >= kn are left alone.
template <int W, int KC, bool SWAP>
__device__ __forceinline__ void stage_panel(double (*dst)[W], MatView const& V, int r0, int q0, int rows, int kn, int lane) {
    if (V.layout == BLASTGPU_PANEL) {
        for (int idx = lane; idx < W * KC; idx += 32) {
            int const r = idx % W, q = idx / W;
            if (q < kn) dst[q][r] = r0 + r < rows ? (SWAP ? V(q0 + q, r0 + r) : V(r0 + r, q0 + q)) : 0.0;
        }
        return;
    }
    int64_t const ld = V.ld;
    if ((V.layout == BLASTGPU_COL_MAJOR) != SWAP) {  // r contiguous
        constexpr int Q = W >= 32 ? 1 : 32 / W, RS = W >= 32 ? W / 32 : 1;  // columns a pass, passes a column
        if constexpr (W % 32 == 0 || 32 % W == 0) {
            int const r = lane % W, q = lane / W;
            double const* p = V.p + r0 + r + (q0 + q) * ld;
#pragma unroll
            for (int s = 0; s < KC / Q; ++s)
#pragma unroll
                for (int h = 0; h < RS; ++h)
                    if (q + s * Q < kn) dst[q + s * Q][r + 32 * h] = r0 + r + 32 * h < rows ? p[s * Q * ld + 32 * h] : 0.0;
        } else {
            for (int idx = lane; idx < W * kn; idx += 32) {
                int const r = idx % W, q = idx / W;
                dst[q][r] = r0 + r < rows ? V.p[r0 + r + (q0 + q) * ld] : 0.0;
            }
        }
    } else if (kn > 8) {  // q contiguous, 16 lanes to a row
        int const q = lane % KC, r = lane / KC;
        double const* p = V.p + q0 + q + (r0 + r) * ld;
        if (q < kn) {
#pragma unroll
            for (int s = 0; s < W / 2; ++s) dst[q][r + 2 * s] = r0 + r + 2 * s < rows ? p[2 * s * ld] : 0.0;
        }
    } else {  // 8 lanes
        int const q = lane % 8, r = lane / 8;
        double const* p = V.p + q0 + q + (r0 + r) * ld;
        if (q < kn) {
#pragma unroll
            for (int s = 0; s < W / 4; ++s) dst[q][r + 4 * s] = r0 + r + 4 * s < rows ? p[4 * s * ld] : 0.0;
        }
    }
}

// An instance's output tiles are dealt out to `parts` warps (1 when the batch fills the chip by itself).
template <int RM, int RN, class Batch>
__global__ void __launch_bounds__(kWarps * 32, kCtas<RM, RN>) gemm_warp_kernel(Batch batch, int64_t count, int parts) {
    constexpr int WM = 4 * RM, WN = 8 * RN, KC = kKChunk;
    __shared__ __align__(16) double sA[kWarps][KC][WM];
    __shared__ __align__(16) double sB[kWarps][KC][WN];

    int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int64_t const w = (int64_t)blockIdx.x * kWarps + warp;
    int64_t const b = parts == 1 ? w : w / parts;
    if (b >= count) return;
    int const part = (int)(w - b * parts);

    int M, N, K;
    double alpha, beta;
    MatView A, B, C, D;
    batch.get(b, M, N, K, alpha, beta, A, B, C, D);

    int const lr = lane & 3, lc = lane >> 2;
    double (*a_s)[WM] = sA[warp];
    double (*b_s)[WN] = sB[warp];

    constexpr bool kEarly = RM * RN <= 4;
    bool const dense = C.layout == BLASTGPU_COL_MAJOR && D.layout == BLASTGPU_COL_MAJOR;
    int const tm = (M + WM - 1) / WM, tn = (N + WN - 1) / WN;
    int mi = part % max(tm, 1), nj = part / max(tm, 1);
    while (nj < tn && tm > 0) {
        int const ti = mi * WM, tj = nj * WN, i0 = ti + lr * RM, j0 = tj + lc * RN;
        double ce[RM][RN];  // C, loaded ahead of the products in small tiles
        if (kEarly && dense) {
#pragma unroll
            for (int c = 0; c < RN; ++c)
#pragma unroll
                for (int r = 0; r < RM; ++r)
                    ce[r][c] = j0 + c < N && i0 + r < M ? C.p[i0 + r + (int64_t)(j0 + c) * C.ld] : 0.0;
        }
        double acc[RM][RN];
#pragma unroll
        for (int r = 0; r < RM; ++r)
#pragma unroll
            for (int c = 0; c < RN; ++c) acc[r][c] = 0.0;

        for (int kc = 0; kc < K; kc += KC) {
            int const kn = min(KC, K - kc);
            __syncwarp();
            stage_panel<WM, KC, false>(a_s, A, ti, kc, M, kn, lane);
            stage_panel<WN, KC, true>(b_s, B, tj, kc, N, kn, lane);
            __syncwarp();
#pragma unroll 4
            for (int q = 0; q < kn; ++q) {
                double av[RM], bv[RN];
#pragma unroll
                for (int r = 0; r < RM; ++r) av[r] = a_s[q][lr * RM + r];
#pragma unroll
                for (int c = 0; c < RN; ++c) bv[c] = b_s[q][lc * RN + c];
#pragma unroll
                for (int c = 0; c < RN; ++c)
#pragma unroll
                    for (int r = 0; r < RM; ++r) acc[r][c] = fma(av[r], bv[c], acc[r][c]);
            }
        }
        // Epilogue: acc *= alpha (exact, and left out, for 1); d = fma(beta, c, acc).
        if (alpha != 1.0) {
#pragma unroll
            for (int c = 0; c < RN; ++c)
#pragma unroll
                for (int r = 0; r < RM; ++r) acc[r][c] *= alpha;
        }
        if (dense) {
            double* d = D.p + i0 + (int64_t)j0 * D.ld;
#pragma unroll
            for (int c = 0; c < RN; ++c)
#pragma unroll
                for (int r = 0; r < RM; ++r)
                    if (j0 + c < N && i0 + r < M) {
                        double const cv = kEarly ? ce[r][c] : C.p[i0 + r + (int64_t)(j0 + c) * C.ld];
                        d[r + (int64_t)c * D.ld] = fma(beta, cv, acc[r][c]);
                    }
        } else {
#pragma unroll
            for (int c = 0; c < RN; ++c)
#pragma unroll
                for (int r = 0; r < RM; ++r)
                    if (j0 + c < N && i0 + r < M) D(i0 + r, j0 + c) = fma(beta, C(i0 + r, j0 + c), acc[r][c]);
        }
        mi += parts;
        while (mi >= tm) mi -= tm, ++nj;
    }
}

template <int RM, int RN, class Batch>
int launch_shape(Batch const& batch, int64_t count, int parts, cudaStream_t stream) {
    int64_t const blocks = (count * parts + kWarps - 1) / kWarps;
    if (blocks > 0x7fffffff) return BLASTGPU_ERR_TOO_LARGE;
    gemm_warp_kernel<RM, RN><<<(unsigned)blocks, kWarps * 32, 0, stream>>>(batch, count, parts);
    return check_launch();
}

// The warp tile (0 = 8 x 8, 1 = 16 x 16, 2 = 24 x 24, 3 = 16 x 8) and whether an instance's tiles go to one
// warp or to a warp each, by the multiply-adds that the busiest scheduler gets. A tile without padding runs
// at 0.83 (8 x 8) to 0.90 (24 x 24) of the binary64 rate, since a larger tile has fewer loads per
// multiply-add, and a warp costs a dozen multiply-adds to start. Padding, and warps that do not divide
// evenly among the schedulers, cost in full. Measured: 24 x 24 x 24 x 10,000 in one tile 255 us, in 8 x 8 tiles
// 278 us; 57 x 39 x 23 x 3,000 in 8 x 8 tiles 354 us, in 24 x 24 453 us; 75 x 66 x 64 x 4,586 in 16 x 8 tiles 2.86 ms,
// in 8 x 8 3.24 ms; one 128 x 128 x 128 a warp a tile 25 us, one warp 4.6 ms. 32 x 32 tiles were never ahead.
struct Choice {
    int shape, parts;
};
Choice choose(int64_t count, int m, int n, int k, int only) {
    static constexpr struct { int wm, wn; double rate; } kShapes[] = {
        {8, 8, 0.83}, {16, 16, 0.87}, {24, 24, 0.90}, {16, 8, 0.845}};
    int64_t const schedulers = 4 * (int64_t)sm_count();
    Choice best{0, 1};
    double cost = 1e300;
    for (int s = 0; s < 4; ++s) {
        if (only >= 0 && s != only) continue;
        int64_t const tiles = (int64_t)((m + kShapes[s].wm - 1) / kShapes[s].wm) * ((n + kShapes[s].wn - 1) / kShapes[s].wn);
        double const tile = kShapes[s].wm * kShapes[s].wn / 32.0 * (k + 2) / kShapes[s].rate;
        for (int split = 0; split < 2; ++split) {
            int64_t const parts = split ? tiles : 1;
            int64_t const rounds = (count * parts + schedulers - 1) / schedulers;
            double const c = rounds * (tile * (tiles / parts) + 12);
            if (c < cost && parts <= 0x7fffffff) cost = c, best = {s, (int)parts};
        }
    }
    return best;
}

template <class Batch>
int launch_gemm(Batch const& batch, int64_t count, int max_m, int max_n, int max_k, cudaStream_t stream) {
    if (count == 0 || max_m == 0 || max_n == 0) return BLASTGPU_SUCCESS;
    if (count > 0x7fffffffll * kWarps) return BLASTGPU_ERR_TOO_LARGE;
    // The autotuner's choice for a square bin, "gemm.shape.m24": sizes that round up to the same multiple of 8.
    int only = -1;
    if ((max_m + 7) / 8 == (max_n + 7) / 8) {
        char key[32];
        snprintf(key, sizeof(key), "gemm.shape.m%d", ((max_m + 7) / 8) * 8);
        only = tune_get(key, -1);
        if (only > 3) only = -1;
    }
    Choice const c = choose(count, max_m, max_n, max_k, only);
    switch (c.shape) {
        case 0: return launch_shape<2, 1>(batch, count, c.parts, stream);
        case 1: return launch_shape<4, 2>(batch, count, c.parts, stream);
        case 2: return launch_shape<6, 3>(batch, count, c.parts, stream);
        default: return launch_shape<4, 1>(batch, count, c.parts, stream);
    }
}

}  // namespace
}  // namespace blastgpu

using namespace blastgpu;

extern "C" {

int blastgpu_dgemm_strided(int trans_a, int trans_b, int m, int n, int k, double alpha,
                           const double* A, int lda, int64_t stride_a,
                           const double* B, int ldb, int64_t stride_b, double beta,
                           const double* C, int ldc, int64_t stride_c,
                           double* D, int ldd, int64_t stride_d,
                           int64_t batch, blastgpu_stream_t stream) {
    if (trans_a != 0 && trans_a != 1) return -1;
    if (trans_b != 0 && trans_b != 1) return -2;
    if (m < 0) return -3;
    if (n < 0) return -4;
    if (k < 0) return -5;
    // Leading dimensions bound the stored arrays: A is m x k (k x m when trans_a), B k x n.
    if (lda < (trans_a ? (k > 0 ? k : 1) : (m > 0 ? m : 1)) && m > 0 && k > 0) return -8;
    if (ldb < (trans_b ? (n > 0 ? n : 1) : (k > 0 ? k : 1)) && n > 0 && k > 0) return -11;
    if (ldc < (m > 0 ? m : 1) && m > 0 && n > 0) return -15;
    if (ldd < (m > 0 ? m : 1) && m > 0 && n > 0) return -18;
    if (batch < 0) return -20;
    if (batch == 0 || m == 0 || n == 0) return BLASTGPU_SUCCESS;
    if (k > 0 && (!A || !B)) return !A ? -7 : -10;
    if (!C) return -14;
    if (!D) return -17;
    StridedGemm g;
    g.m = m; g.n = n; g.k = k; g.alpha = alpha; g.beta = beta;
    g.A = MatView{const_cast<double*>(A), lda, trans_a ? BLASTGPU_ROW_MAJOR : BLASTGPU_COL_MAJOR, 1};
    g.B = MatView{const_cast<double*>(B), ldb, trans_b ? BLASTGPU_ROW_MAJOR : BLASTGPU_COL_MAJOR, 1};
    g.C = MatView{const_cast<double*>(C), ldc, BLASTGPU_COL_MAJOR, 1};
    g.D = MatView{D, ldd, BLASTGPU_COL_MAJOR, 1};
    g.sa = stride_a; g.sb = stride_b; g.sc = stride_c; g.sd = stride_d;
    return launch_gemm(g, batch, m, n, k, as_cuda(stream));
}

int blastgpu_dgemm_bwd_batched(const blastgpu_gemm_bwd_desc* desc, int64_t batch, int max_dim, int32_t* status,
                               blastgpu_stream_t stream) {
    if (batch < 0) return -2;
    if (batch == 0) return BLASTGPU_SUCCESS;
    if (!desc) return -1;
    if (max_dim < 0) return -3;
    int64_t const blocks = (batch + 3) / 4;
    if (blocks > 0x7fffffff) return BLASTGPU_ERR_TOO_LARGE;
    cudaStream_t const s = as_cuda(stream);
    gemm_bwd_c_kernel<<<(unsigned)blocks, 128, 0, s>>>(desc, batch, status);
    int st = check_launch();
    if (st != BLASTGPU_SUCCESS) return st;
    st = launch_gemm(GemmBwdBatch{desc, 0}, batch, max_dim, max_dim, max_dim, s);
    if (st != BLASTGPU_SUCCESS) return st;
    return launch_gemm(GemmBwdBatch{desc, 1}, batch, max_dim, max_dim, max_dim, s);
}

int blastgpu_dgemm_batched(const blastgpu_gemm_desc* desc, int64_t batch, int max_m, int max_n,
                           int max_k, blastgpu_stream_t stream) {
    if (batch < 0) return -2;
    if (batch == 0) return BLASTGPU_SUCCESS;
    if (!desc) return -1;
    if (max_m < 0) return -3;
    if (max_n < 0) return -4;
    if (max_k < 0) return -5;
    DescGemm g{desc};
    return launch_gemm(g, batch, max_m, max_n, max_k, as_cuda(stream));
}

}  // extern "C"
