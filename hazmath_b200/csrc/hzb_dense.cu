// hzb_dense.cu -- coarsest-level dense factorisation (FP64).
//
// The coarsest matrix (<= coarse_dof rows, ~1-2k) is expanded to a dense
// lower triangle and factored A = L L^T, L is inverted, and A^{-1} =
// L^{-T} L^{-1} is formed once, so that every V-cycle applies the coarse
// solve as one dense matrix-vector product (n^2 FP64 reads from L2) instead
// of two dependent triangular sweeps.
//
// The arithmetic (n^3 multiply-adds, 0.3 ms at the FP64 rate for n = 2000) is
// short against the chain of n / 32 panel steps, so the chain is what the
// layout serves: one launch per 32-column step, in which the CTA of the
// first trailing tile also factors and inverts the next diagonal block (it
// alone holds it, updated), and the inverse of L by doubling block sizes
// (2 log2(n / 32) launches of independent tiles) instead of block row by
// block row.  n = 1600: 6.5 -> 2.0 ms; n = 1999: 9.5 -> 2.6 ms.  What bounds a
// step now is shared memory bandwidth while many tiles are left, then the 32
// dependent columns of the diagonal block.
// This file may contract a*b+c into FMA: the coarse solve is a direct
// solve that agrees with the reference's sparse LDL^T only to rounding.
#include <algorithm>
#include "hzb_setup.cuh"

namespace hzb {

constexpr int NB = 32;          // panel width
constexpr int TB = 64;          // tile of the updates and products
constexpr int TK = 16;          // depth of a staged slice of the products

__global__ void k_dense_from_csr(int n, const int *__restrict__ ia,
                                 const int *__restrict__ ja,
                                 const double *__restrict__ a, double *D) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        for (int k = ia[i]; k < ia[i + 1]; ++k) D[(size_t)i * n + ja[k]] += a[k];
}

// Inverse of the Cholesky factor of a 32 x 32 SPD block, by 256 threads:
// elimination in place (below the diagonal the factors of the unit lower
// inverse replace the eliminated entries), then a scaling by the pivots'
// roots.  W: the block (read) and the result; V: a second buffer, the two
// alternate so that a column costs one barrier.  Returns false on a pivot
// that is not positive (every thread sees the same pivots).
using Block = double[NB][NB + 1];
__device__ __forceinline__ bool invert_factor(Block *W, Block *V) {
    const int k = threadIdx.x & 31, w = threadIdx.x >> 5;
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = (*W)[w + 8 * q][k];
    __syncthreads();
    Block *in = W, *out = V;
    for (int j = 0; j < NB; ++j) {
        const double piv = (*in)[j][j];
        if (!(piv > 0.0)) return false;
        const double rp = 1.0 / piv, jk = (*in)[j][k];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = w + 8 * q;
            if (i > j) {
                const double f = (*in)[i][j] * rp;
                v[q] = k == j ? -f : v[q] - f * jk;
            }
            (*out)[i][k] = v[q];
        }
        __syncthreads();
        Block *t = in; in = out; out = t;
    }
    // *in: pivots on the diagonal, the unit lower inverse below it
    double r[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = w + 8 * q;
        const double root = sqrt((*in)[i][i]);
        r[q] = k < i ? (*in)[i][k] / root : k == i ? 1.0 / root : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) (*W)[w + 8 * q][k] = r[q];
    __syncthreads();
    return true;
}

// the block at (r0, r0), padded with the identity, inverted into X
__device__ __forceinline__ void factor_diag(int n, int r0, Block *W, Block *V, double *X,
                                            int *bad) {
    if (!invert_factor(W, V)) {
        if (threadIdx.x == 0) *bad = 1;
        return;
    }
    const int k = threadIdx.x & 31;
    for (int i = threadIdx.x >> 5; i < NB; i += 8)
        if (r0 + i < n && k <= i) X[(size_t)(r0 + i) * n + r0 + k] = (*W)[i][k];
}

__global__ void __launch_bounds__(256)
k_chol_first(int n, const double *__restrict__ D, double *X, int *bad) {
    __shared__ Block W, V;
    const int k = threadIdx.x & 31;
    for (int i = threadIdx.x >> 5; i < NB; i += 8) {
        const int a = max(i, k), b = min(i, k);   // the lower triangle is the one kept
        W[i][k] = a < n ? D[(size_t)a * n + b] : (i == k ? 1.0 : 0.0);
    }
    __syncthreads();
    factor_diag(n, 0, &W, &V, X, bad);
}

// Step j0: the panel L[:, j0:j0+32] = D[:, j0:j0+32] X_JJ^T and the trailing
// update D -= L L^T, one 64 x 64 tile of the lower triangle per CTA.  Every
// tile forms the two panel slices it needs (a third of its arithmetic), so
// panel and update need no launch between them; tiles of the first column
// store theirs.  The first tile goes on to the next diagonal block.
__global__ void __launch_bounds__(256)
k_chol_step(int n, int j0, double *D, double *L, double *X, int *bad) {
    __shared__ double Pi[TB][NB + 1], Pk[TB][NB + 1], Ij[NB][NB + 1];
    if (*(volatile int *)bad) return;
    int bi = (int)((sqrt(8.0 * blockIdx.x + 1.0) - 1.0) * 0.5);
    while ((bi + 1) * (bi + 2) / 2 <= (int)blockIdx.x) ++bi;
    while (bi * (bi + 1) / 2 > (int)blockIdx.x) --bi;
    const int bk = (int)blockIdx.x - bi * (bi + 1) / 2;
    const int r0 = j0 + NB, ri = r0 + bi * TB, rk = r0 + bk * TB;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int i = w; i < TB; i += 8) {
        Pi[i][lane] = ri + i < n ? D[(size_t)(ri + i) * n + j0 + lane] : 0.0;
        if (bi != bk) Pk[i][lane] = rk + i < n ? D[(size_t)(rk + i) * n + j0 + lane] : 0.0;
        if (i < NB) Ij[i][lane] = lane <= i ? X[(size_t)(j0 + i) * n + j0 + lane] : 0.0;
    }
    __syncthreads();
    double li[8], lk[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) li[q] = lk[q] = 0.0;
#pragma unroll 8
    for (int t = 0; t < NB; ++t) {
        const double x = Ij[lane][t];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            li[q] += Pi[w + 8 * q][t] * x;
            if (bi != bk) lk[q] += Pk[w + 8 * q][t] * x;
        }
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int i = w + 8 * q;
        Pi[i][lane] = li[q];
        Pk[i][lane] = bi != bk ? lk[q] : li[q];
        if (bk == 0 && ri + i < n) L[(size_t)(ri + i) * n + j0 + lane] = li[q];
    }
    __syncthreads();
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double acc[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) acc[q][p] = 0.0;
#pragma unroll 8
    for (int t = 0; t < NB; ++t) {
        double a[4], b[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) { a[q] = Pi[ty + 16 * q][t]; b[q] = Pk[tx + 16 * q][t]; }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int p = 0; p < 4; ++p) acc[q][p] += a[q] * b[p];
    }
    const bool next = blockIdx.x == 0;   // this tile holds the next diagonal block
    if (next) __syncthreads();           // Pi becomes its buffers
    Block *W = reinterpret_cast<Block *>(&Pi[0][0]);
    Block *V = reinterpret_cast<Block *>(&Pi[NB][0]);
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int i = ty + 16 * q, k = tx + 16 * p;
            double d = 0.0;
            if (ri + i < n && rk + k <= ri + i) {
                const size_t at = (size_t)(ri + i) * n + rk + k;
                d = D[at] - acc[q][p];
                D[at] = d;
            }
            if (next && i < NB && k <= i) {
                if (ri + i >= n) d = i == k ? 1.0 : 0.0;
                (*W)[i][k] = d;
                (*W)[k][i] = d;
            }
        }
    if (next) {
        __syncthreads();
        factor_diag(n, r0, W, V, X, bad);
    }
}

// One 64 x 64 tile of a product, C(i, c) = sum over k in [k0, k1) of
// a(i, k) b(k, c): 256 threads, 4 x 4 values each, slices of 16 staged in
// shared memory with the next slice's loads in flight.
template <typename FA, typename FB>
__device__ __forceinline__ void tile_product(int k0, int k1, FA fa, FB fb, bool a_by_k,
                                             double acc[4][4]) {
    __shared__ double As[TK][TB + 1], Bs[TK][TB + 1];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) acc[q][p] = 0.0;
    double ra[4], rb[4];
    // a row-major over k (a_by_k false): 16 threads along k; else 64 along i
    const int ai = a_by_k ? (threadIdx.x & 63) : (threadIdx.x >> 4);
    const int ak = a_by_k ? (threadIdx.x >> 6) : (threadIdx.x & 15);
    const int bc = threadIdx.x & 63, bk = threadIdx.x >> 6;
    auto fetch = [&](int kb) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = a_by_k ? ai : ai + 16 * q, k = a_by_k ? ak + 4 * q : ak;
            ra[q] = kb + k < k1 ? fa(i, kb + k) : 0.0;
            rb[q] = kb + bk + 4 * q < k1 ? fb(kb + bk + 4 * q, bc) : 0.0;
        }
    };
    fetch(k0);
    for (int kb = k0; kb < k1; kb += TK) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            As[a_by_k ? ak + 4 * q : ak][a_by_k ? ai : ai + 16 * q] = ra[q];
            Bs[bk + 4 * q][bc] = rb[q];
        }
        __syncthreads();
        if (kb + TK < k1) fetch(kb + TK);
#pragma unroll
        for (int t = 0; t < TK; ++t) {
            double a[4], b[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) { a[q] = As[t][ty + 16 * q]; b[q] = Bs[t][tx + 16 * q]; }
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int p = 0; p < 4; ++p) acc[q][p] += a[q] * b[p];
        }
        __syncthreads();
    }
}

// Doubling step of X = L^{-1} for blocks of s rows, pair blockIdx.z: with
// [L11 0; L21 L22] and X11, X22 known, X21 = -X22 (L21 X11).  half 0 forms
// T = L21 X11, half 1 X21 = -X22 T.
__global__ void __launch_bounds__(256)
k_trinv_pair(int n, int s, int half, const double *__restrict__ L, double *X, double *T) {
    const int r1 = blockIdx.z * 2 * s, r2 = r1 + s;    // block rows 1 and 2
    const int i0 = blockIdx.y * TB, c0 = blockIdx.x * TB;
    const int m = min(s, n - r2);                      // rows of block 2
    if (i0 >= m) return;
    double acc[4][4];
    if (half == 0)   // X11 is lower triangular: k >= c
        tile_product(c0, s,
                     [&](int i, int k) {
                         return i0 + i < m ? L[(size_t)(r2 + i0 + i) * n + r1 + k] : 0.0;
                     },
                     [&](int k, int c) {
                         return c0 + c <= k ? X[(size_t)(r1 + k) * n + r1 + c0 + c] : 0.0;
                     }, false, acc);
    else             // X22 is lower triangular: k <= i
        tile_product(0, min(m, i0 + TB),
                     [&](int i, int k) {
                         return i0 + i < m && k <= i0 + i
                                    ? X[(size_t)(r2 + i0 + i) * n + r2 + k] : 0.0;
                     },
                     [&](int k, int c) {
                         return c0 + c < s ? T[(size_t)(r2 + k) * n + r1 + c0 + c] : 0.0;
                     }, false, acc);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    double *out = half == 0 ? T : X;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int i = i0 + ty + 16 * q, c = c0 + tx + 16 * p;
            if (i < m && c < s)
                out[(size_t)(r2 + i) * n + r1 + c] = half == 0 ? acc[q][p] : -acc[q][p];
        }
}

// Ainv = X^T X, X lower triangular: the tiles of the lower triangle, each
// written twice
__global__ void __launch_bounds__(256)
k_xtx(int n, const double *__restrict__ X, double *Ainv) {
    if (blockIdx.x > blockIdx.y) return;
    const int i0 = blockIdx.y * TB, c0 = blockIdx.x * TB;
    double acc[4][4];
    tile_product(i0, n,   // X[k][i] = 0 for k < i
                 [&](int i, int k) {
                     return i0 + i <= k ? X[(size_t)k * n + i0 + i] : 0.0;
                 },
                 [&](int k, int c) {
                     return c0 + c <= k ? X[(size_t)k * n + c0 + c] : 0.0;
                 }, true, acc);
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            const int i = i0 + ty + 16 * q, c = c0 + tx + 16 * p;
            if (i < n && c <= i) {
                Ainv[(size_t)i * n + c] = acc[q][p];
                Ainv[(size_t)c * n + i] = acc[q][p];
            }
        }
}

int dense_inverse(const DCsr<double> &A, double **Ainv_out, cudaStream_t s) {
    const int n = A.n;
    *Ainv_out = nullptr;
    // D: the trailing matrix, then the products of the doubling steps;
    // Ainv holds L until the inverse of L is complete
    double *D = nullptr, *X = nullptr, *Ainv = nullptr;
    int *bad = nullptr;
    const size_t nn = (size_t)n * n;
    int rc = SUCCESS, hbad = 0;
    cudaError_t e;
    if ((rc = dalloc(&D, nn))) goto done;
    if ((rc = dalloc(&X, nn))) goto done;
    if ((rc = dalloc(&Ainv, nn))) goto done;
    if ((rc = dalloc(&bad, 1))) goto done;
    cudaMemsetAsync(D, 0, nn * sizeof(double), s);
    cudaMemsetAsync(bad, 0, sizeof(int), s);
    k_dense_from_csr<<<grid_for(n), 256, 0, s>>>(n, A.ia, A.ja, A.val, D);
    k_chol_first<<<1, 256, 0, s>>>(n, D, X, bad);
    count_launch(2);
    for (int j0 = 0; j0 + NB < n; j0 += NB) {
        const int nt = div_up(n - j0 - NB, TB);
        k_chol_step<<<nt * (nt + 1) / 2, 256, 0, s>>>(n, j0, D, Ainv, X, bad);
        count_launch();
    }
    for (int b = NB; b < n; b *= 2) {
        const int pairs = div_up(n - b, 2 * b), t = div_up(b, TB);
        for (int half = 0; half < 2; ++half)
            k_trinv_pair<<<dim3(t, t, pairs), 256, 0, s>>>(n, b, half, Ainv, X, D);
        count_launch(2);
    }
    k_xtx<<<dim3(div_up(n, TB), div_up(n, TB)), 256, 0, s>>>(n, X, Ainv);
    count_launch();
    e = cudaMemcpyAsync(&hbad, bad, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto done; }
    if (hbad) { set_error_msg("coarse matrix is not positive definite"); rc = ERROR_DATA_ZERODIAG; goto done; }
    *Ainv_out = Ainv;
    Ainv = nullptr;
done:
    dfree(D); dfree(X); dfree(Ainv); dfree(bad);
    return rc;
}

}  // namespace hzb
