// hzb_gs.cu -- exact Gauss-Seidel over small level sets, streamed.
//
// A level set of the lexicographic order depends on the one before it, so what
// bounds a sweep is the time from one set to the next.  One CTA runs the sets
// in order and keeps everything a set needs in shared memory: the matrix rows
// are stored a second time in the schedule's order (a set's rows of one length,
// filled up with zeros against a place that holds zero, the diagonal left out), x, b and the diagonals are put
// into that order before the sweep and x back after it, so that a warp of its
// own copies whole groups of sets ahead by a few contiguous bulk copies.  x
// lies in a ring indexed by place in the schedule, wide enough that every
// entry's value is in it: new values of earlier sets, the old iterate for
// later ones.  A set is then one barrier, the shared loads of x (a thread has
// its row's first entries in registers by then) and the chain of subtractions.
//   Measured on the sets of 2D 5-point levels: 0.47 us a set with loads
// rotated through registers and x in shared memory, 1.3 with x in global
// memory (gathers of just written values miss L1), 0.7 to 1.3 with
// asynchronous 8-byte gathers in place of the permuted vectors (along an
// anti-diagonal each touches a line of its own, and they fill the queue that
// the shared loads of the computing warps go through), 0.6 with a set's copies
// issued inside its barrier, 0.6 with a test per entry (200 instructions a set,
// each waiting for the one before), 0.27 to 0.35 with one set's loads behind the
// other's, 0.18 to 0.23 now that parts of the CTA take the sets in turn.
//   The row sum runs in CSR order from b_i with the diagonal skipped, each
// value rounded as in gs_rows: the same bits.
#include "hzb_gs_plan.h"
#include "hzb_solver.cuh"
#include <algorithm>
#include <type_traits>

namespace hzb {

namespace {

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes,
                                          unsigned long long *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
                 "[%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)), "l"(src), "r"(bytes),
                 "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void bar_init(unsigned long long *bar, unsigned count) {
    asm volatile("mbarrier.init.shared.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// wait for the phase of the given parity; bounded: a copy that never arrives
// is reported, and nobody waits any more
__device__ __forceinline__ void bar_wait(unsigned long long *bar, unsigned parity, int *dead,
                                         int *err) {
    unsigned done = 0;
    for (unsigned spin = 0; !done; ++spin) {
        asm volatile("{\n.reg .pred p;\n"
                     "mbarrier.try_wait.parity.shared.b64 p, [%1], %2;\n"
                     "selp.u32 %0, 1, 0, p;\n}"
                     : "=r"(done) : "r"(smem_u32(bar)), "r"(parity) : "memory");
        if (done || *(volatile int *)dead) return;
        if (spin > (1u << 20)) {
            *(volatile int *)dead = 1;
            atomicExch(err, 1);
            return;
        }
    }
}

// What a sweep runs on; group: sets per stage, E and R a stage's capacity.
struct GsSweep {
    const int4 *info;
    const unsigned short *col;
    const double *val;
    const double2 *bd;
    double *x;
    int ns, group, E, R, stages, ring, dist, places, skip_place;
};

// A thread's row of a set with Z entries: loaded before the barrier that
// completes the previous set, finished behind it.
template <int Z>
struct GsRow {
    unsigned c[Z / 2];              // two ring places each
    double v[Z];
    // pairs of values `step` pairs apart
    __device__ __forceinline__ void load(const unsigned short *col, const double *val,
                                         int step = 1) {
        if (Z == 8) {
            const uint4 u = *reinterpret_cast<const uint4 *>(col);
            c[0] = u.x;
            c[1] = u.y;
            c[2 % (Z / 2)] = u.z;
            c[3 % (Z / 2)] = u.w;
        } else if (Z % 4 == 0) {
#pragma unroll
            for (int q = 0; q < Z / 4; ++q) {
                const uint2 u = reinterpret_cast<const uint2 *>(col)[q];
                c[2 * q] = u.x;
                c[2 * q + 1] = u.y;
            }
        } else {
#pragma unroll
            for (int q = 0; q < Z / 2; ++q) c[q] = reinterpret_cast<const unsigned *>(col)[q];
        }
#pragma unroll
        for (int q = 0; q < Z / 2; ++q) {
            const double2 u = reinterpret_cast<const double2 *>(val)[q * step];
            v[2 * q] = u.x;
            v[2 * q + 1] = u.y;
        }
    }
    __device__ __forceinline__ void gather(const double *ring, double *x) const {
#pragma unroll
        for (int q = 0; q < Z / 2; ++q) {
            x[2 * q] = ring[c[q] & 0xffffu];
            x[2 * q + 1] = ring[c[q] >> 16];
        }
    }
    __device__ __forceinline__ double finish(const double *x, double acc) const {
#pragma unroll
        for (int q = 0; q < Z; ++q) acc -= v[q] * x[q];
        return acc;
    }
    __device__ __forceinline__ double sum(const double *ring, double acc) const {
        double x[Z];
        gather(ring, x);
        return finish(x, acc);
    }
};

template <int KIND, int UZ>
__global__ void __launch_bounds__((UZ ? GS_TURNS : 1) * GS_ROWS + 32, 1)
k_gs_stream(const __grid_constant__ GsSweep A, double w, int *err) {
    extern __shared__ __align__(16) unsigned char smem[];
    int4 *info = reinterpret_cast<int4 *>(smem);
    double *ring = reinterpret_cast<double *>(info + A.ns);   // and a place that holds zero
    unsigned char *stage0 = reinterpret_cast<unsigned char *>(ring + A.ring + 2);
    const int stage_bytes = (int)gs_stage(A.E, A.R);
    unsigned long long *full =
        reinterpret_cast<unsigned long long *>(stage0 + A.stages * stage_bytes);
    unsigned long long *empty = full + A.stages;
    __shared__ int s_dead;
    // threads that compute, and those of them on one set
    const int ns = A.ns, t = threadIdx.x, all = blockDim.x - 32, nt = UZ ? all / GS_TURNS : all;
    for (int k = t; k < ns; k += blockDim.x) info[k] = A.info[k];
    if (t == 0) {
        s_dead = 0;
        ring[A.ring] = 0.0;
        for (int k = 0; k < A.stages; ++k) {
            bar_init(full + k, 1);
            bar_init(empty + k, 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    if (t >= all) {
        // groups of sets into their stages, and x as far as their rows reach
        if (t > all) return;
        int loaded = 0, to = 0, k = 0;  // places of x copied or on their way; the stage
        unsigned parity = 1;            // the first round finds every stage empty
        for (int s0 = 0; s0 < ns; s0 += A.group) {
            const int4 I0 = info[s0], I1 = info[min(s0 + A.group, ns) - 1];
            const int rows = gs_end_place(I1) - I0.x, e = gs_end_entry(I1) - I0.w;
            int upto = (gs_end_place(I1) + A.dist + GS_BLOCK - 1) / GS_BLOCK * GS_BLOCK;
            upto = max(min(upto, A.places), loaded);
            bar_wait(empty + k, parity, &s_dead, err);
            double *val = reinterpret_cast<double *>(stage0 + k * stage_bytes);
            double2 *bd = reinterpret_cast<double2 *>(val + A.E);
            unsigned short *col = reinterpret_cast<unsigned short *>(bd + A.R);
            const unsigned bytes = (unsigned)(e * 10 + rows * 16 + (upto - loaded) * 8);
            asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;"
                         ::"r"(smem_u32(full + k)), "r"(bytes) : "memory");
            if (e) {
                bulk_copy(val, A.val + I0.w, e * 8, full + k);
                bulk_copy(col, A.col + I0.w, e * 2, full + k);
            }
            bulk_copy(bd, A.bd + I0.x, rows * 16, full + k);
            for (; loaded < upto; loaded += GS_BLOCK) {   // the ring is a multiple of GS_BLOCK
                bulk_copy(ring + to, A.x + loaded, GS_BLOCK * 8, full + k);
                to = to + GS_BLOCK == A.ring ? 0 : to + GS_BLOCK;
            }
            if (++k == A.stages) {
                k = 0;
                parity ^= 1u;
            }
        }
        return;
    }
    const int val_bytes = A.E * 8, col_at = val_bytes + A.R * 16;
    auto store = [&](const int4 &I, int row, double acc, double dinv) {
        if (row >= gs_rows(I)) return;
        const int place = I.x + row, at = I.z + row;
        double *px = ring + (at < A.ring ? at : at - A.ring);
        if (KIND == 0) {
            const double xn = acc * dinv;
            *px = xn;
            A.x[place] = xn;
        } else if (place != A.skip_place && fabs(dinv) > double(SMALLREAL)) {
            const double xn = KIND == 1 ? w * (acc / dinv) + (1 - w) * *px : acc / dinv;
            *px = xn;
            A.x[place] = xn;
        }
    };
    if constexpr (UZ > 0) {
        // Three parts of the CTA take the sets in turn: a part loads its next set
        // (370 cycles) while the others finish one each (190, and 70 for the
        // barrier), so that between two sets lie a barrier, the loads of x and
        // the sums only.
        const int turn = t / nt, row = t - turn * nt, warp0 = row & ~31;
        int in = turn, k = 0;           // the set's place in its group, the group's stage
        unsigned parity = 0;
        auto place = [&]() {
            while (in >= A.group) {
                in -= A.group;
                if (++k == A.stages) {
                    k = 0;
                    parity ^= 1u;
                }
            }
        };
        GsRow<UZ> r;
        double2 bd = make_double2(0.0, 0.0);
        int4 I = make_int4(0, 0, 0, 0);
        auto fetch = [&](int s) {
            I = info[s];
            if (warp0 >= gs_rows(I)) return;
            bar_wait(full + k, parity, &s_dead, err);
            const int4 F = info[s - in];
            const unsigned char *stage = stage0 + k * stage_bytes;
            const int at = row < gs_rows(I) ? row : 0;   // idle threads load the first row
            const double *val = reinterpret_cast<const double *>(stage) + (I.w - F.w);
            const unsigned short *col =
                reinterpret_cast<const unsigned short *>(stage + col_at) + (I.w - F.w);
            r.load(col + at * UZ, val + 2 * at, gs_pitch(gs_rows(I)));
            bd = reinterpret_cast<const double2 *>(stage + val_bytes)[I.x - F.x + at];
        };
        place();
        if (turn < ns) fetch(turn);
        for (int s = turn; s < ns; s += GS_TURNS) {
            // the set before is complete, and its group when this set begins one
            __syncwarp();
            if (s) asm volatile("bar.sync %0, %1;" ::"r"(1 + turn), "r"(2 * nt) : "memory");
            if (in == 0 && s && row == 0)
                asm volatile("mbarrier.arrive.shared.b64 _, [%0];"
                             ::"r"(smem_u32(empty + (k ? k : A.stages) - 1)) : "memory");
            if (warp0 < gs_rows(I)) {
                double x[UZ];
                r.gather(ring, x);
                store(I, row, r.finish(x, bd.x), bd.y);
            }
            // what this part wrote to the ring in a group comes before the copies
            // that replace it
            if (in + GS_TURNS >= A.group) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (s + 1 < ns)
                asm volatile("bar.arrive %0, %1;" ::"r"(1 + (turn + 1) % GS_TURNS), "r"(2 * nt) : "memory");
            in += GS_TURNS;
            place();
            if (s + GS_TURNS < ns) fetch(s + GS_TURNS);
        }
    } else {
        int k = 0, in_group = 0;        // the stage at hand, sets of it begun
        unsigned parity = 0;
        int e0 = 0, x0 = 0;             // the group's first entry and place
        const unsigned char *stage = stage0;
        unsigned long long *release = nullptr;   // the stage that the next barrier frees
        // the previous set is complete, and its group when this set begins one
        auto barrier = [&]() {
            asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory");
            if (release && t == 0)
                asm volatile("mbarrier.arrive.shared.b64 _, [%0];" ::"r"(smem_u32(release))
                             : "memory");
        };
        for (int s = 0; s < ns; ++s) {
            const int4 I = info[s];
            if (in_group == 0) {
                bar_wait(full + k, parity, &s_dead, err);
                x0 = I.x;
                e0 = I.w;
                stage = stage0 + k * stage_bytes;
            }
            const int Z = gs_width(I);
            const bool on = t < gs_rows(I);
            const int at = on ? I.w - e0 + t * Z : 0;   // idle threads load the first row
            const double *val = reinterpret_cast<const double *>(stage) + at;
            const unsigned short *col =
                reinterpret_cast<const unsigned short *>(stage + col_at) + at;
            const double2 bd =
                reinterpret_cast<const double2 *>(stage + val_bytes)[on ? I.x - x0 + t : 0];
            double acc;
            switch (Z) {   // the same for every thread
            case 0: barrier(); acc = bd.x; break;
            case 2: { GsRow<2> r; r.load(col, val); barrier(); acc = r.sum(ring, bd.x); break; }
            case 4: { GsRow<4> r; r.load(col, val); barrier(); acc = r.sum(ring, bd.x); break; }
            case 6: { GsRow<6> r; r.load(col, val); barrier(); acc = r.sum(ring, bd.x); break; }
            case 8: { GsRow<8> r; r.load(col, val); barrier(); acc = r.sum(ring, bd.x); break; }
            default: {
                barrier();
                acc = bd.x;
                for (int u = 0; u < Z; u += 2) {
                    GsRow<2> r;
                    r.load(col + u, val + u);
                    acc = r.sum(ring, acc);
                }
            }
            }
            release = nullptr;
            store(I, t, acc, bd.y);
            if (++in_group == A.group) {
                // what this group wrote to the ring comes before the copies that
                // replace it
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                in_group = 0;
                release = empty + k;
                if (++k == A.stages) {
                    k = 0;
                    parity ^= 1u;
                }
            }
        }
    }
}

// Place of entry u of a set's row t: with one width for all sets its pairs lie
// side by side with the other rows' (a warp's loads are then free of conflicts),
// else with the row's own.
__device__ __forceinline__ int gs_at(int uniform, int pitch, int Z, int t, int u) {
    return uniform ? (u / 2 * pitch + t) * 2 + u % 2 : t * Z + u;
}

// vectors into the schedule's order (src: row of a place, -1 for padding)
__global__ void k_gs_in(int places, const int *__restrict__ src, const double *__restrict__ b,
                        const double *__restrict__ d, const double *__restrict__ x, double2 *bd,
                        double *xp) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < places; q += gridDim.x * blockDim.x) {
        const int i = src[q];
        bd[q] = i >= 0 ? make_double2(b[i], d[i]) : make_double2(0.0, 0.0);
        xp[q] = i >= 0 ? x[i] : 0.0;
    }
}
// The same for a matrix in the caller's arrays, whose values are read as they
// are: the rows' values go into the schedule's order too (a CTA per set).
__global__ void __launch_bounds__(GS_ROWS)
k_gs_in_values(int places, const int4 *__restrict__ info, int uniform,
               const int *__restrict__ src, const double *__restrict__ b,
               const double *__restrict__ d, const double *__restrict__ x,
               const int *__restrict__ ia, const int *__restrict__ ja,
               const double *__restrict__ a, double2 *bd, double *xp, double *val) {
    const int4 I = info[blockIdx.x];
    const int t = threadIdx.x, pitch = gs_pitch(gs_rows(I)), Z = gs_width(I);
    if (t < pitch) {
        constexpr int W = 8;        // entries in flight
        const int i = src[I.x + t];
        const int k0 = i >= 0 ? ia[i] : 0, k1 = i >= 0 ? ia[i + 1] : 0;
        bd[I.x + t] = i >= 0 ? make_double2(b[i], d[i]) : make_double2(0.0, 0.0);
        xp[I.x + t] = i >= 0 ? x[i] : 0.0;
        int u = 0;
        for (int kb = k0; kb < k1; kb += W) {
            int c[W];
            double v[W];
#pragma unroll
            for (int q = 0; q < W; ++q) {
                c[q] = kb + q < k1 ? ja[kb + q] : i;
                v[q] = kb + q < k1 ? a[kb + q] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < W; ++q)
                if (c[q] != i) val[I.w + gs_at(uniform, pitch, Z, t, u++)] = v[q];
        }
    }
    if (blockIdx.x == gridDim.x - 1)    // up to a whole block of places
        for (int q = gs_end_place(I) + t; q < places; q += GS_ROWS) {
            bd[q] = make_double2(0.0, 0.0);
            xp[q] = 0.0;
        }
}
__global__ void k_gs_out(int places, const int *__restrict__ src, const double *__restrict__ xp,
                         double *x) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < places; q += gridDim.x * blockDim.x) {
        const int i = src[q];
        if (i >= 0) x[i] = xp[q];
    }
}

// one CTA per set: its rows in ascending order to their places (neighbouring
// rows lie side by side in the ring then), and the longest row without the
// diagonal, made even
__global__ void __launch_bounds__(GS_ROWS)
k_gs_place(const int *__restrict__ rows, const int *__restrict__ set_ptr,
           const int *__restrict__ start, const int *__restrict__ ia, const int *__restrict__ ja,
           int *src, int *place, int *width) {
    __shared__ int r[GS_ROWS], sh[32];
    const int s = blockIdx.x, t = threadIdx.x;
    const int q0 = set_ptr[s], m = set_ptr[s + 1] - q0;
    const int i = t < m ? rows[q0 + t] : 0x7fffffff;
    r[t] = i;
    __syncthreads();
    int len = 0;
    if (t < m) {
        int rank = 0;
        for (int q = 0; q < m; ++q) rank += r[q] < i;
        src[start[s] + rank] = i;
        place[i] = start[s] + rank;
        for (int k = ia[i]; k < ia[i + 1]; ++k) len += ja[k] != i;
    }
    len = block_max(len, sh);
    if (t == 0) width[s] = (len + 1) / 2 * 2;
}

// the largest distance in places between a row and one of its columns
__global__ void k_gs_dist(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                          const int *__restrict__ place, int *dist) {
    __shared__ int sh[32];
    int m = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int p = place[i];
        for (int k = ia[i]; k < ia[i + 1]; ++k) m = max(m, abs(place[ja[k]] - p));
    }
    m = block_max(m, sh);
    if (threadIdx.x == 0) atomicMax(dist, m);
}

// one CTA per set: the entries row by row, zeros against the ring's zero place
// behind a shorter row (subtracting +0.0 * 0.0 changes nothing)
__global__ void __launch_bounds__(GS_ROWS)
k_gs_fill(const int4 *__restrict__ info, int ring, int uniform, const int *__restrict__ src,
          const int *__restrict__ place, const int *__restrict__ ia, const int *__restrict__ ja,
          const double *__restrict__ a, unsigned short *col, double *val) {
    const int4 I = info[blockIdx.x];
    const int t = threadIdx.x, Z = gs_width(I);
    if (t >= gs_pitch(gs_rows(I))) return;
    const int i = t < gs_rows(I) ? src[I.x + t] : -1;
    const int pitch = gs_pitch(gs_rows(I));
    col += I.w + t * Z;
    val += I.w;
    int u = 0;
    if (i >= 0)
        for (int k = ia[i]; k < ia[i + 1]; ++k) {
            const int j = ja[k];
            if (j == i) continue;
            col[u] = (unsigned short)(place[j] % ring);
            val[gs_at(uniform, pitch, Z, t, u)] = a[k];
            ++u;
        }
    for (; u < Z; ++u) {
        col[u] = (unsigned short)ring;
        val[gs_at(uniform, pitch, Z, t, u)] = 0.0;
    }
}

}  // namespace

void GsStream::release() {
    dfree(info);
    dfree(src);
    dfree(place);
    dfree(col);
    dfree(val);
    dfree(bd);
    dfree(xp);
    stages = 0;
}

int gs_stream_build(const DCsr<double> &A, Schedule *sc, cudaStream_t s) {
    GsStream &G = sc->stream;
    G.release();
    const int n = A.n, ns = (int)sc->h_ptr.size() - 1;
    // sets of at most a row per thread throughout, and few enough of them
    std::vector<int> start;
    const int places = gs_places(sc->h_ptr, &start);
    if (!places) return SUCCESS;
    std::vector<int> width(ns);
    int *d_start = nullptr, *d_width = nullptr, dist = 0;
    int rc = SUCCESS;
    cudaError_t e = cudaSuccess;
    auto done = [&](bool keep) {
        dfree(d_start);
        dfree(d_width);
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; }
        if (rc || !keep) G.release();
        return rc;
    };
    if ((rc = dalloc(&d_start, ns)) || (rc = dalloc(&d_width, ns + 1)) ||
        (rc = dalloc(&G.src, places)) || (rc = dalloc(&G.place, n)))
        return done(false);
    e = cudaMemcpyAsync(d_start, start.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(G.src, 0xff, sizeof(int) * places, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(d_width + ns, 0, sizeof(int), s);
    if (e != cudaSuccess) return done(false);
    k_gs_place<<<ns, GS_ROWS, 0, s>>>(sc->rows, sc->set_ptr, d_start, A.ia, A.ja, G.src, G.place,
                                      d_width);
    k_gs_dist<<<grid_for(n), 256, 0, s>>>(n, A.ia, A.ja, G.place, d_width + ns);
    count_launch(2);
    e = cudaMemcpyAsync(width.data(), d_width, sizeof(int) * ns, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&dist, d_width + ns, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return done(false);
    const GsPlan P = gs_plan(sc->h_ptr, start, places, width, dist);
    if (!P.stages) return done(false);
    int max_rows = 0;
    for (int k = 0; k < ns; ++k) max_rows = std::max(max_rows, sc->h_ptr[k + 1] - sc->h_ptr[k]);
    if ((rc = dalloc(&G.info, ns)) || (rc = dalloc(&G.col, P.ents)) || (rc = dalloc(&G.val, P.ents)) ||
        (rc = dalloc(&G.bd, places)) || (rc = dalloc(&G.xp, places)))
        return done(false);
    e = cudaMemcpyAsync(G.info, P.info.data(), sizeof(int4) * ns, cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) {
        k_gs_fill<<<ns, GS_ROWS, 0, s>>>(G.info, P.ring, P.uniform, G.src, G.place, A.ia, A.ja, A.val,
                                         G.col, G.val);
        count_launch();
        e = cudaMemcpyAsync(&G.last_place, G.place + n - 1, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);   // and the host arrays above
    }
    G.ns = ns;
    G.uniform = P.uniform;
    G.threads = (max_rows + 31) / 32 * 32;
    G.group = P.group;
    G.E = P.E;
    G.R = P.R;
    G.ring = P.ring;
    G.stages = P.stages;
    G.dist = dist;
    G.places = places;
    return done(true);
}

int gs_stream_sweep(const Schedule &sc, const DCsr<double> *live, const double *d,
                    const double *b, double *x, int kind, double w, int *err, cudaStream_t s) {
    const GsStream &G = sc.stream;
    const int skip_place = (kind & GS_SKIP_LAST) ? G.last_place : -1;   // SGS leaves row n - 1
    auto of_kind = [&](auto k) {
        constexpr int K = decltype(k)::value;
        switch (G.uniform) {
        case 2: return k_gs_stream<K, 2>;
        case 4: return k_gs_stream<K, 4>;
        case 6: return k_gs_stream<K, 6>;
        case 8: return k_gs_stream<K, 8>;
        default: return k_gs_stream<K, 0>;
        }
    };
    const int K = kind & 15;
    auto kernel = K == 0   ? of_kind(std::integral_constant<int, 0>())
                  : K == 1 ? of_kind(std::integral_constant<int, 1>())
                           : of_kind(std::integral_constant<int, 2>());
    HZB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)GS_SMEM));
    if (live)
        k_gs_in_values<<<G.ns, GS_ROWS, 0, s>>>(G.places, G.info, G.uniform, G.src, b, d, x,
                                                live->ia, live->ja, live->val, G.bd, G.xp, G.val);
    else
        k_gs_in<<<grid_for(G.places), 256, 0, s>>>(G.places, G.src, b, d, x, G.bd, G.xp);
    const GsSweep A = {G.info, G.col, G.val, G.bd, G.xp, G.ns, G.group, G.E, G.R, G.stages,
                       G.ring, G.dist, G.places, skip_place};
    kernel<<<1, G.threads * (G.uniform ? GS_TURNS : 1) + 32, gs_smem(G.ns, G.E, G.R, G.ring, G.stages), s>>>(A, w, err);
    k_gs_out<<<grid_for(G.places), 256, 0, s>>>(G.places, G.src, G.xp, x);
    count_launch(3);
    HZB_LAUNCH_CHECK();
    return SUCCESS;
}

}  // namespace hzb
