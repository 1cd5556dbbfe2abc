// hzb_small.cu -- the l1-Jacobi V-cycle on its small levels.
//
// A small level (SMALL_ROWS_32, SMALL_NNZ_64: some hundred thousand rows) lies in
// L2, and a kernel lasts as long as its launch and its chain of dependent loads:
// row pointers, columns, x, at 0.3 to 0.4 us each (2.4 us a node of the graph in
// all on the smallest).  So here
// work is merged where a row's result is all the next step needs of it: the
// residual is formed for the fine rows of a coarse row and summed at once,
// with the coarse level's first sweep from x = 0 (b_i / d_i) behind it, and
// the last sweep of a level adds its result to the finer level's x, which
// leaves pre + post kernels per level instead of pre + post + 3 (+ 1 in FP64,
// which zeroes x).  And every kernel is launched programmatically: it starts
// while its predecessor runs, loads what is constant of its row (pointers,
// columns, values, norms) into registers, and waits for the predecessor only
// then, with the gathers of x left to do.
//   One cooperative kernel for all these levels was slower (5 us a phase, 4.6
// with the rows in registers or shared memory): the barrier costs 1.2 us and
// empties L1.
//
// FP64: one thread per row sums in CSR order and every value is rounded as by
// the separate kernels, so the cycle's result is theirs bit for bit.  FP32:
// LPR lanes share a row.
#include "hzb_solver.cuh"
#include <algorithm>

namespace hzb {

namespace {

constexpr int SMALL_BLOCK = 256;

template <typename T>
struct SmallLevel {
    int n, nc;
    const int *ia, *ja;
    const T *val, *d;               // d: l1 row norms
    const int *ria, *rja;           // fine rows of the next level's rows
    T *b, *x[2];                    // x[0]: the pre-smoother's first buffer
    const float *omega;
};

// the finer level a result is added to (x null: none)
template <typename T>
struct SmallUp {
    const int *ria, *rja;
    T *x;
};

// Programmatic launch: let the next kernel of the stream start, and wait for
// the previous one (and its writes).  What the kernels load before the wait is
// written by none of them.
__device__ __forceinline__ void launch_next() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void wait_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A row at hand: its entries' range, and the first B entries of this lane
// (entry q of lane `sub` is k0 + q LPR with k0 = ia[i] + sub; col -1: none).
template <typename T, int LPR, int B>
struct SmallRow {
    int k0, k1;
    int c[B];
    T v[B];
    __device__ __forceinline__ void load(const SmallLevel<T> &L, int i, int sub) {
        k0 = __ldg(L.ia + i) + sub;
        k1 = __ldg(L.ia + i + 1);
#pragma unroll
        for (int q = 0; q < B; ++q) {
            const int k = k0 + q * LPR;
            c[q] = k < k1 ? __ldg(L.ja + k) : -1;
            v[q] = k < k1 ? __ldg(L.val + k) : T(0);
        }
    }
    // t -= a x (MINUS) or t += a x over the lane's entries, in order
    template <bool MINUS>
    __device__ __forceinline__ T sum(const SmallLevel<T> &L, const T *x, T t) const {
        T xv[B];
#pragma unroll
        for (int q = 0; q < B; ++q) xv[q] = c[q] >= 0 ? x[c[q]] : T(0);
#pragma unroll
        for (int q = 0; q < B; ++q)
            if (c[q] >= 0) t = MINUS ? t - v[q] * xv[q] : t + v[q] * xv[q];
        constexpr int R = 4;    // the rest of a longer row
        for (int kb = k0 + B * LPR; kb < k1; kb += R * LPR) {
            T vr[R], xr[R];
#pragma unroll
            for (int q = 0; q < R; ++q) {
                const int k = kb + q * LPR;
                vr[q] = k < k1 ? __ldg(L.val + k) : T(0);
                xr[q] = k < k1 ? x[__ldg(L.ja + k)] : T(0);
            }
#pragma unroll
            for (int q = 0; q < R; ++q)
                if (kb + q * LPR < k1) t = MINUS ? t - vr[q] * xr[q] : t + vr[q] * xr[q];
        }
        return t;
    }
};

template <typename T, int LPR>
__device__ __forceinline__ T small_lanes_sum(T t) {
#pragma unroll
    for (int o = LPR / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o, LPR);
    return t;
}

// x_i after the first sweep from x = 0
template <typename T>
__device__ __forceinline__ T small_first(T d, const float *omega, int i, T b) {
    T xi = T(0);
    if (fabs(d) > T(SMALLREAL)) xi += (omega ? T(omega[i]) : T(1)) * (b / d);
    return xi;
}

// Into the first level: b = R w (w null: b is there), and its first sweep.
template <typename T>
__global__ void __launch_bounds__(SMALL_BLOCK)
k_small_first(const __grid_constant__ SmallLevel<T> L, const T *w, const int *__restrict__ ria,
              const int *__restrict__ rja) {
    launch_next();
    const int i = blockIdx.x * SMALL_BLOCK + threadIdx.x;
    const bool on = i < L.n;
    const T d = on ? __ldg(L.d + i) : T(0);
    const int k0 = on && w ? __ldg(ria + i) : 0, k1 = on && w ? __ldg(ria + i + 1) : 0;
    wait_previous();
    if (!on) return;
    T t = T(0);
    if (w) {
        for (int k = k0; k < k1; ++k) t += w[__ldg(rja + k)];
        L.b[i] = t;
    } else {
        t = L.b[i];
    }
    L.x[0][i] = small_first(d, L.omega, i, t);
}

// One sweep x -> xn; with U.x the result is added to the finer level instead.
template <typename T, int LPR, int B>
__global__ void __launch_bounds__(SMALL_BLOCK)
k_small_sweep(const __grid_constant__ SmallLevel<T> L, const T *x, T *xn,
              const __grid_constant__ SmallUp<T> U) {
    launch_next();
    const int sub = LPR == 1 ? 0 : threadIdx.x % LPR;
    const int g = (blockIdx.x * SMALL_BLOCK + threadIdx.x) / LPR;
    const int i = min(g, L.n - 1);
    const bool on = g < L.n;
    SmallRow<T, LPR, B> row;
    row.load(L, i, sub);
    const T d = __ldg(L.d + i);
    const float om = L.omega ? __ldg(L.omega + i) : 0.f;
    int u0 = 0, u1 = 0, up = -1;
    if (U.x && on) {
        u0 = __ldg(U.ria + i) + sub;
        u1 = __ldg(U.ria + i + 1);
        if (u0 < u1) up = __ldg(U.rja + u0);
    }
    wait_previous();
    const T xu = up >= 0 ? U.x[up] : T(0);
    T xi = x[i];
    T t = row.template sum<true>(L, x, sub == 0 ? L.b[i] : T(0));
    t = small_lanes_sum<T, LPR>(t);
    if (fabs(d) > T(SMALLREAL)) {
        if (L.omega) xi += T(om) * (t / d);
        else xi += t / d;
    }
    if (!on) return;
    if (!U.x) {
        if (sub == 0) xn[i] = xi;
        return;
    }
    if (up >= 0) U.x[up] = xu + (T(0) + xi);
    for (int k = u0 + LPR; k < u1; k += LPR) {
        const int j = __ldg(U.rja + k);
        U.x[j] = U.x[j] + (T(0) + xi);
    }
}

// Residual of the fine rows of a coarse row, summed: the coarse b; with `first`
// the coarse level's first sweep.
template <typename T, int LPR, int B>
__global__ void __launch_bounds__(SMALL_BLOCK)
k_small_restrict(const __grid_constant__ SmallLevel<T> L, const T *x, T *cb, T *cx,
                 const T *__restrict__ cd) {
    launch_next();
    const int sub = LPR == 1 ? 0 : threadIdx.x % LPR;
    const int g = (blockIdx.x * SMALL_BLOCK + threadIdx.x) / LPR;
    const int c = min(g, L.nc - 1);
    const int q0 = __ldg(L.ria + c), q1 = __ldg(L.ria + c + 1);
    int i[2];
    SmallRow<T, LPR, B> row[2];     // most coarse rows have two
#pragma unroll
    for (int q = 0; q < 2; ++q) i[q] = q0 + q < q1 ? __ldg(L.rja + q0 + q) : -1;
#pragma unroll
    for (int q = 0; q < 2; ++q)
        if (i[q] >= 0) row[q].load(L, i[q], sub);
    const T d = cx ? __ldg(cd + c) : T(0);
    wait_previous();
    auto one = [&](const SmallRow<T, LPR, B> &r, int k, T t) {
        const T bi = L.b[k];
        if (LPR == 1) return t + (bi - r.template sum<false>(L, x, T(0)));
        return r.template sum<true>(L, x, sub == 0 ? t + bi : t);
    };
    T t = T(0);
    if (i[0] >= 0) t = one(row[0], i[0], t);
    if (i[1] >= 0) t = one(row[1], i[1], t);
    for (int q = q0 + 2; q < q1; ++q) {
        const int k = __ldg(L.rja + q);
        row[0].load(L, k, sub);
        t = one(row[0], k, t);
    }
    t = small_lanes_sum<T, LPR>(t);
    if (g < L.nc && sub == 0) {
        cb[c] = t;
        if (cx) cx[c] = small_first<T>(d, nullptr, c, t);
    }
}

// Coarsest level: a warp per row of the dense inverse, whose first entries are
// loaded before the wait; the result goes to the finer level.
template <typename T>
__global__ void __launch_bounds__(SMALL_BLOCK)
k_small_coarse(int n, const double *__restrict__ Ainv, const T *b,
               const __grid_constant__ SmallUp<T> U) {
    launch_next();
    constexpr int G = 16;
    const int lane = threadIdx.x & 31;
    const int r = (blockIdx.x * SMALL_BLOCK + threadIdx.x) >> 5;
    if (r >= n) return;
    const double *row = Ainv + (size_t)r * n;
    double m[G];
#pragma unroll
    for (int q = 0; q < G; ++q) m[q] = lane + 32 * q < n ? __ldg(row + lane + 32 * q) : 0.0;
    const int u0 = __ldg(U.ria + r) + lane, u1 = __ldg(U.ria + r + 1);
    wait_previous();
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < G; ++q)
        if (lane + 32 * q < n) t += m[q] * (double)b[lane + 32 * q];
#pragma unroll 8
    for (int c = lane + 32 * G; c < n; c += 32) t += __ldg(row + c) * (double)b[c];
    t = warp_sum(t);
    const T xi = T(0) + (T)t;
    for (int k = u0; k < u1; k += 32) {
        const int j = __ldg(U.rja + k);
        U.x[j] = U.x[j] + xi;
    }
}

template <typename T>
struct SmallData;
template <>
struct SmallData<float> {
    static constexpr int LPR = 4, B = 4;
    static bool fits(const Level &L) {
        return L.n <= SMALL_ROWS_32 && L.largest_agg <= SMALL_AGG;
    }
    static const int *ia(const Level &L) { return L.ia32; }
    static const int *ja(const Level &L) { return L.ja32; }
    static const float *val(const Level &L) { return L.val32; }
    static const float *d(const Level &L) { return L.l1_32; }
    static float *b(const Level &L) { return L.b32; }
    static float *x(const Level &L) { return L.x32; }
    static float *w(const Level &L) { return L.w32; }
    static float *t(const Level &L) { return L.t32; }
};
template <>
struct SmallData<double> {
    static constexpr int LPR = 1, B = 8;
    static bool fits(const Level &L) {
        return L.nnz <= SMALL_NNZ_64 && (long long)SMALL_ROW_64 * L.n >= L.nnz &&
               L.largest_agg <= SMALL_AGG;
    }
    static const int *ia(const Level &L) { return L.ia; }
    static const int *ja(const Level &L) { return L.ja; }
    static const double *val(const Level &L) { return L.val; }
    static const double *d(const Level &L) { return L.l1_64; }
    static double *b(const Level &L) { return L.b; }
    static double *x(const Level &L) { return L.x; }
    static double *w(const Level &L) { return L.w; }
    static double *t(const Level &L) { return L.t; }
};

template <typename K, typename... Args>
int small_launch(K kernel, long long threads, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(std::max(1, div_up(threads, SMALL_BLOCK)));
    cfg.blockDim = dim3(SMALL_BLOCK);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    HZB_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
    count_launch();
    return SUCCESS;
}

}  // namespace

template <typename T>
int small_first_level(const hzb_solver *S, const AMG_param &cyc, int l0, bool zero) {
    using D = SmallData<T>;
    const int nl = S->nl;
    const bool jac = sizeof(T) == 4 && cyc.smoother == SMOOTHER_JACOBI;   // the FP32 cycle's one sweep
    if (S->batch || cyc.cycle_type != V_CYCLE || (cyc.smoother != SMOOTHER_L1DIAG && !jac) ||
        cyc.presmooth_iter < 1 || cyc.postsmooth_iter < 1 || cyc.coarse_scaling == ON ||
        !S->Ainv || (sizeof(T) == 8 && cyc.coarse_solver != SOLVER_UMFPACK))
        return nl;
    int l = nl - 1;
    while (l > l0 && D::fits(S->lv[l - 1]) && !S->lv[l - 1].sa &&
           (l - 1 > l0 || zero) && D::d(S->lv[l - 1]))
        --l;
    return l < nl - 1 ? l : nl;
}

template <typename T>
int small_levels(hzb_solver *S, int lb, int l0, const AMG_param &cyc) {
    using D = SmallData<T>;
    constexpr int LPR = D::LPR, B = D::B;
    const int last = S->nl - 1, pre = cyc.presmooth_iter, post = cyc.postsmooth_iter;
    cudaStream_t s = S->s;
    auto level = [&](int l) {
        const Level &L = S->lv[l];
        SmallLevel<T> t;
        t.n = L.n;
        t.nc = L.nc;
        t.ia = D::ia(L);
        t.ja = D::ja(L);
        t.val = D::val(L);
        t.d = D::d(L);
        t.ria = L.ria;
        t.rja = L.rja;
        t.b = D::b(L);
        // the first buffer such that the last sweep ends in x
        const int swap = (pre - 1 + post) & 1;
        t.x[swap] = D::x(L);
        t.x[swap ^ 1] = D::t(L);
        t.omega = l == 0 && S->omega_active ? S->omega : nullptr;
        return t;
    };
    const SmallUp<T> none = {nullptr, nullptr, nullptr};
    // the finer level under level l, and its x when level l is done
    auto up = [&](int l) {
        if (l == l0) return none;
        const Level &F = S->lv[l - 1];
        return SmallUp<T>{F.ria, F.rja, l > lb ? level(l - 1).x[(pre - 1) & 1] : D::x(F)};
    };
    {
        const SmallLevel<T> L = level(lb);
        const Level *F = lb > l0 ? &S->lv[lb - 1] : nullptr;
        HZB_TRY(small_launch(k_small_first<T>, L.n, s, L, F ? (const T *)D::w(*F) : nullptr,
                             (const int *)(F ? F->ria : nullptr),
                             (const int *)(F ? F->rja : nullptr)));
    }
    for (int l = lb; l < last; ++l) {
        const SmallLevel<T> L = level(l), C = level(l + 1);
        for (int j = 1; j < pre; ++j)
            HZB_TRY(small_launch(k_small_sweep<T, LPR, 2 * B>, (long long)L.n * LPR, s, L,
                                 (const T *)L.x[(j - 1) & 1], L.x[j & 1], none));
        HZB_TRY(small_launch(k_small_restrict<T, LPR, B>, (long long)L.nc * LPR, s, L,
                             (const T *)L.x[(pre - 1) & 1], C.b, l + 1 < last ? C.x[0] : nullptr,
                             C.d));
    }
    {
        const SmallLevel<T> C = level(last);
        HZB_TRY(small_launch(k_small_coarse<T>, 32LL * C.n, s, C.n, (const double *)S->Ainv,
                             (const T *)C.b, up(last)));
    }
    for (int l = last - 1; l >= lb; --l) {
        const SmallLevel<T> L = level(l);
        for (int j = 0; j < post; ++j) {
            const int from = (pre - 1 + j) & 1;
            // the last result is only needed a level up, or as the answer
            HZB_TRY(small_launch(k_small_sweep<T, LPR, 2 * B>, (long long)L.n * LPR, s, L,
                                 (const T *)L.x[from], L.x[from ^ 1],
                                 j == post - 1 ? up(l) : none));
        }
    }
    return SUCCESS;
}

template int small_first_level<float>(const hzb_solver *, const AMG_param &, int, bool);
template int small_first_level<double>(const hzb_solver *, const AMG_param &, int, bool);
template int small_levels<float>(hzb_solver *, int, int, const AMG_param &);
template int small_levels<double>(hzb_solver *, int, int, const AMG_param &);

}  // namespace hzb
