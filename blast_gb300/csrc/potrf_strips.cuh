// Binary64 Cholesky factorisation by a group of T threads, for the matrices, or their last columns, that the
// fixed-point kernels leave to binary64 (fix64.cuh).
//
// Reference: blast::potrf (dense/Potrf.hpp:20-106): strips of 4 columns; an element takes the fused products of all
// earlier columns in ascending order, then its strip's.
#pragma once

#include "common.cuh"

namespace blastgpu {

// Columns from .. n-1 (from a multiple of 4): src(r, c) are the matrix's entries, dst(r, c) the factor's, whose
// columns before `from` are there (the two may be one). In columns from .. given-1 the diagonal block is there too,
// and the rows without todo(r). diag: 16 doubles that the group shares; sync(): its barrier. Returns 0 or the first
// pivot that is not positive + 1.
// The multiply-adds bound it (2 a clock and SM), a thread's rows one after another: loads come from L1 and L2.
template <int T, class Src, class Dst, class Todo, class Sync>
__device__ __noinline__ int potrf_strips(int n, int from, int given, Src src, Dst dst, Todo todo, double* diag, int tid,
                                         Sync sync) {
    int info = 0;
    for (int k = from; k < n; k += 4) {
        int const nc = min(4, n - k);
        bool const have = k < given;
        double d[4][4], y[4];
        if (have) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
#pragma unroll
                for (int j = 0; j < c; ++j) d[c][j] = dst(k + c, k + j);
                y[c] = rcp_nr(dst(k + c, k + c));
            }
        }
        for (int r0 = k; r0 < n; r0 += T) {
            int const r = r0 + tid;
            bool const mine = r < n && (!have || todo(r));
            double acc[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[c] = mine && c < nc && r >= k + c ? src(r, k + c) : 0.0;
            if (mine) {
#pragma unroll 4
                for (int l = 0; l < k; ++l) {
                    double const a = dst(r, l);
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[c] = fma(-a, dst(k + min(c, nc - 1), l), acc[c]);
                }
            }
            if (r0 == k && !have) {  // the diagonal block, in every thread
                if (tid < nc) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) diag[4 * tid + c] = acc[c];
                }
                sync();
#pragma unroll
                for (int q = 0; q < 4; ++q)
#pragma unroll
                    for (int c = 0; c <= q; ++c) d[q][c] = q < nc ? diag[4 * q + c] : 0.0;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (c < nc) {
#pragma unroll
                        for (int j = 0; j < c; ++j)
#pragma unroll
                            for (int q = c; q < 4; ++q) d[q][c] = fma(-d[c][j], d[q][j], d[q][c]);
                        double const s = d[c][c];
                        if (!(s > 0.0) && info == 0) info = k + c + 1;
                        y[c] = rsqrt_nr(s);
#pragma unroll
                        for (int q = c; q < 4; ++q) d[q][c] *= y[c];
                    }
                }
            }
            if (mine) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    if (c < nc) {
#pragma unroll
                        for (int j = 0; j < c; ++j) acc[c] = fma(-d[c][j], acc[j], acc[c]);
                        acc[c] *= y[c];
                        if (r >= k + c) dst(r, k + c) = acc[c];
                    }
                }
            }
        }
        sync();
    }
    return info;
}

}  // namespace blastgpu
