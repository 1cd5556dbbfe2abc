// hzb_sell.cu -- the sliced-ELL schedule.
//
// A matrix is also kept as 32-row slices, each as wide as its longest row; rows
// are ordered by length (descending, ties by index) inside each 256-row window,
// so the rows of a slice have nearly equal lengths.  Entries 2p and 2p + 1 of a
// row lie side by side, at val[32 (first + 2p) + 2 (slot mod 32)], the last of
// an odd width alone in its line of 32, so the threads of a warp, one row each,
// read their entries with coalesced loads -- no shared-memory staging (full
// occupancy) and no lanes to combine.  Each row's entries keep their CSR order
// and one thread sums them in that order; a row shorter than its slice adds
// zeros times its own last column's x.
//   The sweeps are bound by the memory, so what counts is the bytes of an
// entry: its column is held in 16 bits above the smallest column of its slice
// at its position (base, the same words for the whole warp), which covers any
// matrix whose neighbouring rows reach to similar places; a slice where some
// range is wider keeps 32-bit columns.  A row's index and length share a word.
// 6 bytes an FP32 entry instead of 8, and no test per entry: 222 -> 185 us a
// sweep of 16.6 million rows of up to 7 entries, 150 -> 131 on the next level.
// All 64 warps of an SM have to run for it (32 registers; 221 us with 48 of them);
// fetching entries into L2 some waves ahead gave nothing, several windows a CTA 4 %
// here and a loss on smaller levels.
#include "hzb_setup.cuh"
#include <climits>
#include <type_traits>

namespace hzb {

namespace {
constexpr int SELL_WIN = 256;   // rows sorted together (one CTA)
constexpr int SELL_C = 32;      // rows per slice
constexpr unsigned SELL_ROW = SELL_WIN - 1;   // a slot's row within its window; the length above

template <typename T> struct SellPair;
template <> struct SellPair<float> { using type = float2; };
template <> struct SellPair<double> { using type = double2; };

// One CTA per window: slot of each row by its rank (longer first, then by
// index; rows past n last) and, a warp per slice, its width (the first slot
// holds the longest row), half of it rounded up, and the lines of 64 bytes of
// its columns: the width, or twice that where a position's columns span more
// than 16 bits.
__global__ void __launch_bounds__(SELL_WIN)
k_sell_order(int n, const int *__restrict__ ia, const int *__restrict__ ja, unsigned *slot,
             int *width, int *pairs, int *lines, unsigned long long *total) {
    __shared__ __align__(16) int key[SELL_WIN];
    __shared__ int len[SELL_WIN], row[SELL_WIN], sum[3];
    const int t = threadIdx.x, w0 = blockIdx.x * SELL_WIN;
    const int i = w0 + t;
    const int li = i < n ? ia[i + 1] - ia[i] : -1;
    // length, then index: one compare a pair of rows, four rows a load
    const int k = min(li, INT_MAX / SELL_WIN - 1) * SELL_WIN + (SELL_WIN - 1 - t);
    key[t] = k;
    len[t] = li;
    if (t < 3) sum[t] = 0;
    __syncthreads();
    int rank = 0;
#pragma unroll 8
    for (int q = 0; q < SELL_WIN / 4; ++q) {
        const int4 o = reinterpret_cast<const int4 *>(key)[q];
        rank += (o.x > k) + (o.y > k) + (o.z > k) + (o.w > k);
    }
    row[rank] = t;
    if (li >= INT_MAX / SELL_WIN) atomicAdd(total, 1ull << 40);   // no room for the length
    slot[w0 + rank] = (unsigned)t | (unsigned)max(li, 0) * SELL_WIN;
    __syncthreads();
    const int r = row[t], l = max(len[r], 0);
    const int k0 = l > 0 ? ia[w0 + r] : 0;
    const int w = __shfl_sync(0xffffffffu, l, 0);
    bool wide = false;
    for (int u = 0; u < w; ++u) {
        const int c = l > 0 ? ja[k0 + min(u, l - 1)] : -1;
        const int lo = __reduce_min_sync(0xffffffffu, c < 0 ? INT_MAX : c);
        const int hi = __reduce_max_sync(0xffffffffu, c);
        wide |= hi - lo > 0xffff;
    }
    if (t % SELL_C == 0) {
        const int sl = (w0 + t) / SELL_C, np = (w + 1) / 2, nl = wide ? 2 * w : w;
        width[sl] = w;
        pairs[sl] = np;
        lines[sl] = nl;
        atomicAdd(sum, w);
        atomicAdd(sum + 1, np);
        atomicAdd(sum + 2, nl);
    }
    __syncthreads();
    if (t < 3) atomicAdd(total + t, (unsigned long long)sum[t]);
}

// entry u's place in a slice of width w: two side by side, the last of an odd width
// alone
__device__ __forceinline__ int sell_at(int u, int w, int lane) {
    return u + 1 == w && u % 2 == 0 ? u * SELL_C + lane : u / 2 * 2 * SELL_C + 2 * lane + u % 2;
}

// A warp per slice: its entries, columns and bases, and its head: first line of
// entries, first line of columns (negated and less one where they are 32 bits
// wide), first pair of bases, width.
__global__ void __launch_bounds__(SELL_WIN)
k_sell_fill(const int *__restrict__ first, const int *__restrict__ pairs,
            const int *__restrict__ lines, const unsigned *__restrict__ slot,
            const int *__restrict__ ia, const int *__restrict__ ja, const float *__restrict__ a,
            int4 *head, unsigned short *col, int2 *base, float *val) {
    const int t = blockIdx.x * SELL_WIN + threadIdx.x, s = t / SELL_C, lane = t % SELL_C;
    const unsigned sl = slot[t];
    const int len = (int)(sl / SELL_WIN);
    const int f0 = first[s], w = first[s + 1] - f0, l0 = lines[s], p0 = pairs[s];
    const bool wide = lines[s + 1] - l0 != w;
    const int k0 = len > 0 ? ia[blockIdx.x * SELL_WIN + (sl & SELL_ROW)] : 0;
    if (lane == 0) head[s] = make_int4(f0, wide ? -l0 - 1 : l0, p0, w);
    for (int u = 0; u < w; ++u) {
        int c = len > 0 ? ja[k0 + min(u, len - 1)] : INT_MAX;
        const int lo = __reduce_min_sync(0xffffffffu, c);
        if (len == 0) c = lo;
        const int at = sell_at(u, w, lane);
        if (val) val[(size_t)f0 * SELL_C + at] = u < len ? a[k0 + u] : 0.f;
        if (lane == 0) reinterpret_cast<int *>(base + p0 + u / 2)[u % 2] = lo;
        unsigned short *q = col + (size_t)l0 * SELL_C;
        if (wide) reinterpret_cast<int *>(q)[at] = c;
        else q[at] = (unsigned short)(c - lo);
    }
}

// The FP64 values of a copy whose FP32 ones are there.
__global__ void __launch_bounds__(SELL_WIN)
k_sell_values(const __grid_constant__ SellView<double> V, const int *__restrict__ ia,
              const double *__restrict__ a, double *val) {
    const int t = blockIdx.x * SELL_WIN + threadIdx.x, lane = t % SELL_C;
    const unsigned sl = V.slot[t];
    const int4 h = V.head[t / SELL_C];
    const int len = (int)(sl / SELL_WIN);
    const int k0 = len > 0 ? ia[blockIdx.x * SELL_WIN + (sl & SELL_ROW)] : 0;
    for (int u = 0; u < h.w; ++u) val[(size_t)h.x * SELL_C + sell_at(u, h.w, lane)] =
        u < len ? a[k0 + u] : 0.0;
}

// W entries of a row, all their loads and gathers in flight at once.  L1: t -= v x
// and d += |v| (t starts at b_i); else t += v x.  val, col and base point at the
// slice's next entries, lane is the thread's.
template <typename T, bool L1, bool WIDE, int W>
__device__ __forceinline__ void sell_entries(const T *__restrict__ val,
                                             const unsigned short *__restrict__ col,
                                             const int2 *__restrict__ base, int lane,
                                             const T *__restrict__ x, T &t, T &d) {
    using V2 = typename SellPair<T>::type;
    T v[W], xv[W];
    int c[W];
#pragma unroll
    for (int q = 0; q < W / 2; ++q) {
        const V2 u = __ldcs(reinterpret_cast<const V2 *>(val) + q * SELL_C + lane);
        v[2 * q] = u.x;
        v[2 * q + 1] = u.y;
        if (WIDE) {
            const int2 k = __ldcs(reinterpret_cast<const int2 *>(col) + q * SELL_C + lane);
            c[2 * q] = k.x;
            c[2 * q + 1] = k.y;
        } else {
            const unsigned k = __ldcs(reinterpret_cast<const unsigned *>(col) + q * SELL_C + lane);
            const int2 b = __ldg(base + q);
            c[2 * q] = b.x + (int)(k & 0xffffu);
            c[2 * q + 1] = b.y + (int)(k >> 16);
        }
    }
    if (W % 2) {
        v[W - 1] = __ldcs(val + (W - 1) * SELL_C + lane);
        c[W - 1] = WIDE ? __ldcs(reinterpret_cast<const int *>(col) + (W - 1) * SELL_C + lane)
                        : __ldg(&base[W / 2].x) + (int)__ldcs(col + (W - 1) * SELL_C + lane);
    }
#pragma unroll
    for (int q = 0; q < W; ++q) xv[q] = __ldg(x + c[q]);
#pragma unroll
    for (int q = 0; q < W; ++q) {
        if (L1) {
            t -= v[q] * xv[q];
            d += fabs(v[q]);
        } else {
            t += v[q] * xv[q];
        }
    }
}

// entries in flight, of FP64 rows half as many (they take twice the registers)
template <typename T> constexpr int SELL_G = sizeof(T) == 8 ? 4 : 8;
template <typename T, bool L1, bool WIDE>
__device__ __forceinline__ void sell_slice(const SellView<T> &V, int4 h, int lane,
                                           const T *__restrict__ x, T &t, T &d) {
    const T *val = V.val + (size_t)h.x * SELL_C;
    const unsigned short *col = V.col + (size_t)(WIDE ? -h.y - 1 : h.y) * SELL_C;
    const int2 *base = V.base + h.z;
    int w = h.w;
    constexpr int G = SELL_G<T>;
    for (; w >= G; w -= G) {
        sell_entries<T, L1, WIDE, G>(val, col, base, lane, x, t, d);
        val += G * SELL_C;
        col += G * SELL_C * (WIDE ? 2 : 1);
        base += G / 2;
    }
    switch (w) {                   // the same for the whole warp
    case 1: sell_entries<T, L1, WIDE, 1>(val, col, base, lane, x, t, d); break;
    case 2: sell_entries<T, L1, WIDE, 2>(val, col, base, lane, x, t, d); break;
    case 3: sell_entries<T, L1, WIDE, 3>(val, col, base, lane, x, t, d); break;
    case 4: if (G > 4) sell_entries<T, L1, WIDE, 4>(val, col, base, lane, x, t, d); break;
    case 5: if (G > 5) sell_entries<T, L1, WIDE, 5>(val, col, base, lane, x, t, d); break;
    case 6: if (G > 6) sell_entries<T, L1, WIDE, 6>(val, col, base, lane, x, t, d); break;
    case 7: if (G > 7) sell_entries<T, L1, WIDE, 7>(val, col, base, lane, x, t, d); break;
    }
}

// Row sum of slot r's row in CSR order.
template <typename T, bool L1>
__device__ __forceinline__ void sell_row(const SellView<T> &V, int r, const T *__restrict__ x,
                                         T &t, T &d) {
    const int4 h = __ldg(V.head + r / SELL_C);
    if (h.y >= 0) sell_slice<T, L1, false>(V, h, r % SELL_C, x, t, d);
    else sell_slice<T, L1, true>(V, h, r % SELL_C, x, t, d);
}

// The sums of this thread's row once more, t on from where it is, over the row's
// own entries only: a zero that fills up a shorter row may meet an infinite or
// NaN x, and the row's own result need not be NaN then.  For the rows whose sum
// came out NaN.  Where it can be it is a call behind the store, the kernel's last
// act, for which nothing is kept in registers: inline the FP64 sweep of 1.8
// million rows took 53 to 55 us, so it takes 49.9 (49.7 without any of this).
template <typename T, bool L1>
__device__ __forceinline__ void sell_row_own(const SellView<T> &V, const T *__restrict__ x, T &t,
                                             T &d) {
    const int r = blockIdx.x * SELL_WIN + threadIdx.x;
    const unsigned sl = __ldcg(V.slot + r);
    const int4 h = __ldcg(V.head + r / SELL_C);
    const unsigned short *col = V.col + (size_t)(h.y < 0 ? -h.y - 1 : h.y) * SELL_C;
#pragma unroll 1
    for (int u = 0; u < (int)(sl / SELL_WIN); ++u) {
        const int at = sell_at(u, h.w, r % SELL_C);
        const int2 b = V.base[h.z + u / 2];
        const int c = h.y < 0 ? reinterpret_cast<const int *>(col)[at]
                              : (u % 2 ? b.y : b.x) + (int)col[at];
        const T v = V.val[(size_t)h.x * SELL_C + at];
        if (L1) {
            t -= v * x[c];
            d += fabs(v);
        } else {
            t += v * x[c];
        }
    }
}

// the sweep's row, from the start
template <typename T>
__device__ __noinline__ void l1_sell_again(const SellView<T> &V, const T *b, const T *x, T *xn,
                                           const float *omega) {
    const int k = blockIdx.x * SELL_WIN +
                  (int)(__ldcg(V.slot + blockIdx.x * SELL_WIN + threadIdx.x) & SELL_ROW);
    T t = b[k], d = T(0), xi = x[k];
    sell_row_own<T, true>(V, x, t, d);
    if (fabs(d) > T(SMALLREAL)) xi += omega ? T(omega[k]) * (t / d) : t / d;
    xn[k] = xi;
}

template <typename T>
__global__ void __launch_bounds__(SELL_WIN, 8)
k_l1_sell(int n, const __grid_constant__ SellView<T> V, const T *__restrict__ b,
          const T *__restrict__ x, T *__restrict__ xn, const float *__restrict__ omega) {
    const int r = blockIdx.x * SELL_WIN + threadIdx.x;
    const unsigned sl = __ldcs(V.slot + r);
    const int i = blockIdx.x * SELL_WIN + (int)(sl & SELL_ROW);
    if (i >= n) return;
    T t = __ldcs(b + i), d = T(0);
    sell_row<T, true>(V, r, x, t, d);
    T xi = x[i];
    if (fabs(d) > T(SMALLREAL)) xi += omega ? T(omega[i]) * (t / d) : t / d;
    xn[i] = xi;
    if (t != t) l1_sell_again<T>(V, b, x, xn, omega);
}

// the product's row, from the start: b_i - A x (RES) or A x
template <typename T, bool RES>
__device__ __noinline__ void spmv_sell_again(const SellView<T> &V, const T *x, T bi, T *yi) {
    T t = T(0), d = T(0);
    sell_row_own<T, false>(V, x, t, d);
    *yi = RES ? bi - t : t;
}

// 64 warps an SM here too (FP64, 16.6 million rows, with (x, y): 290 us; 322 with
// 48, 443 with 32; 364 staged).  SPMV_Y_DOT: the partial sums of (x, y) over the same groups of `rows`
// rows, added in the same order, as the staged kernels (the same bits).
template <typename T, int MODE>
__global__ void __launch_bounds__(SELL_WIN, 8)
k_spmv_sell(int n, const __grid_constant__ SellView<T> V, const T *__restrict__ x,
            const T *__restrict__ b, T *__restrict__ y, T alpha, T *__restrict__ part,
            int rows) {
    const int r = blockIdx.x * SELL_WIN + threadIdx.x;
    const unsigned sl = __ldcs(V.slot + r);
    const int i = blockIdx.x * SELL_WIN + (int)(sl & SELL_ROW);
    if (MODE != SPMV_Y_DOT && i >= n) return;
    const T bi = MODE == SPMV_RES ? __ldcs(b + i) : T(0);
    T t = T(0), d = T(0);
    sell_row<T, false>(V, r, x, t, d);
    if ((MODE == SPMV_AXPY || MODE == SPMV_Y_DOT) && t != t) {
        t = T(0);
        sell_row_own<T, false>(V, x, t, d);
    }
    if (MODE == SPMV_RES) {
        y[i] = bi - t;
        if (t != t) spmv_sell_again<T, true>(V, x, bi, y + i);
    } else if (MODE == SPMV_AXPY) {
        if (alpha == T(1)) y[i] += t;
        else if (alpha == T(-1)) y[i] -= t;
        else y[i] += t * alpha;
    } else if (MODE == SPMV_Y) {
        y[i] = t;
        if (t != t) spmv_sell_again<T, false>(V, x, T(0), y + i);
    } else {
        __shared__ T prod[SELL_WIN], sh[SELL_WIN / 32];
        if (i < n) {
            y[i] = t;
            d = t * __ldg(x + i);
        }
        prod[sl & SELL_ROW] = d;
        __syncthreads();
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, per = rows / 32;
        d = warp_sum(prod[threadIdx.x]);
        if (lane == 0) sh[warp] = d;
        __syncthreads();
        if (warp < SELL_WIN / rows) {
            d = warp_sum(lane < per ? sh[warp * per + lane] : T(0));
            const long long g = (long long)blockIdx.x * (SELL_WIN / rows) + warp;
            if (lane == 0 && g * rows < n) part[g] = d;
        }
    }
}
}  // namespace

int sell_pad_rows(int n) { return (n + SELL_WIN - 1) / SELL_WIN * SELL_WIN; }

int sell_build(int n, const int *ia, const int *ja, const float *a, SellArrays *out,
               cudaStream_t s) {
    *out = SellArrays();
    if (n <= 0) return SUCCESS;
    const int npad = sell_pad_rows(n), nsl = npad / SELL_C, win = npad / SELL_WIN;
    int *cnt = nullptr, *ptr = nullptr, *tmp = nullptr;   // widths, pairs, lines; their sums
    unsigned long long *dtot = nullptr, htot[3] = {0, 0, 0};
    SellArrays S;
    S.npad = npad;
    int rc = SUCCESS;
    if ((rc = dalloc(&S.slot, npad)) || (rc = dalloc(&S.head, nsl)) ||
        (rc = dalloc(&cnt, 3 * (size_t)nsl)) || (rc = dalloc(&ptr, 3 * ((size_t)nsl + 1))) ||
        (rc = dalloc(&tmp, scan_tmp_size(nsl + 1))) || (rc = dalloc(&dtot, 3)))
        goto done;
    if (cudaMemsetAsync(dtot, 0, sizeof(htot), s) != cudaSuccess) {
        rc = ERROR_SOLVER_MISC;
        goto done;
    }
    k_sell_order<<<win, SELL_WIN, 0, s>>>(n, ia, ja, S.slot, cnt, cnt + nsl, cnt + 2 * (size_t)nsl,
                                          dtot);
    count_launch();
    if (cudaMemcpyAsync(htot, dtot, sizeof(htot), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
        rc = ERROR_SOLVER_MISC;
        goto done;
    }
    // a level whose padded slices would not fit an int index, or whose rows a
    // slot's length, gets no copy (the bundles and lanes kernels serve it)
    if (htot[0] * SELL_C > (unsigned long long)(INT_MAX / 2)) goto done;
    for (int q = 0; q < 3 && !rc; ++q)
        rc = scan_exclusive(cnt + (size_t)q * nsl, ptr + q * ((size_t)nsl + 1), nsl, tmp, s);
    if (rc || (a && (rc = dalloc(&S.val, std::max(1ull, htot[0] * SELL_C)))) ||
        (rc = dalloc(&S.base, std::max(1ull, htot[1]))) ||
        (rc = dalloc(&S.col, std::max(1ull, htot[2] * SELL_C))))
        goto done;
    k_sell_fill<<<win, SELL_WIN, 0, s>>>(ptr, ptr + nsl + 1, ptr + 2 * ((size_t)nsl + 1),
                                            S.slot, ia, ja, a, S.head, S.col, S.base, S.val);
    count_launch();
    if (cudaGetLastError() != cudaSuccess) {
        rc = ERROR_SOLVER_MISC;
        goto done;
    }
    S.nval = (size_t)htot[0] * SELL_C;
    *out = S;
done:
    dfree(cnt);
    dfree(ptr);
    dfree(tmp);
    dfree(dtot);
    if (!out->npad) S.release();
    return rc;
}
int sell_values64(SellArrays *S, const int *ia, const double *a, cudaStream_t s) {
    HZB_TRY(dalloc(&S->val64, std::max<size_t>(1, S->nval)));
    k_sell_values<<<S->npad / SELL_WIN, SELL_WIN, 0, s>>>(S->view64(), ia, a, S->val64);
    count_launch();
    HZB_LAUNCH_CHECK();
    return SUCCESS;
}

void SellArrays::release() {
    dfree(slot);
    dfree(head);
    dfree(base);
    dfree(col);
    dfree(val);
    dfree(val64);
    npad = 0;
}

template <typename T>
int sell_l1_sweep(const DCsr<T> &A, const T *b, const T *x, T *xn, const float *omega,
                  cudaStream_t s) {
    k_l1_sell<T><<<A.sell.npad / SELL_WIN, SELL_WIN, 0, s>>>(A.n, A.sell, b, x, xn, omega);
    count_launch();
    HZB_LAUNCH_CHECK();
    return SUCCESS;
}
template int sell_l1_sweep<float>(const DCsr<float> &, const float *, const float *, float *,
                                  const float *, cudaStream_t);
template int sell_l1_sweep<double>(const DCsr<double> &, const double *, const double *,
                                   double *, const float *, cudaStream_t);

template <typename T>
int sell_spmv(const DCsr<T> &A, int mode, const T *x, const T *b, T *y, T alpha, T *part,
              cudaStream_t s) {
    auto go = [&](auto kernel) {
        kernel<<<A.sell.npad / SELL_WIN, SELL_WIN, 0, s>>>(A.n, A.sell, x, b, y, alpha, part,
                                                           A.bundle_rows);
    };
    switch (mode) {
    case SPMV_RES: go(k_spmv_sell<T, SPMV_RES>); break;
    case SPMV_AXPY: go(k_spmv_sell<T, SPMV_AXPY>); break;
    case SPMV_Y_DOT: go(k_spmv_sell<T, SPMV_Y_DOT>); break;
    default: go(k_spmv_sell<T, SPMV_Y>); break;
    }
    count_launch();
    HZB_LAUNCH_CHECK();
    return SUCCESS;
}
template int sell_spmv<float>(const DCsr<float> &, int, const float *, const float *, float *,
                              float, float *, cudaStream_t);
template int sell_spmv<double>(const DCsr<double> &, int, const double *, const double *,
                               double *, double, double *, cudaStream_t);

}  // namespace hzb
