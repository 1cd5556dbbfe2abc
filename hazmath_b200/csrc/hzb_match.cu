// hzb_match.cu -- deterministic parallel matching (fast mode).
//
//   PM_LEAD rounds of mutual choice: every free vertex points at its heaviest
//   free neighbour and mutual pairs match; then red/blue handshake rounds (a
//   hashed coin splits the free vertices, a red vertex proposes to its
//   heaviest free blue neighbour, a blue vertex accepts its heaviest proposer)
//   until a few rounds in a row form no pair.  Leftovers join their first
//   aggregated neighbour.  Mutual choice alone stalls on chains of ever
//   heavier edges (smooth coefficient fields); the handshake alone pairs a
//   vertex only with a neighbour of the other colour, which on the 128^3
//   log-normal problem (sigma 1) left coarser levels and 43 instead of the
//   reference's 38 iterations; a few mutual rounds first gave 39.
//
// Three launches per level: the diagonal, the strong off-diagonal entries of
// every row compacted in place of the row (FP32 weights, no graph of its own,
// so no count, scan and fill), and one cooperative kernel for all rounds, the
// leftovers and the numbering.  A round had been eight launches (three of them
// a scan that numbered its pairs) and a host read, which bound every level
// below a million rows, and each round swept all vertices.  Pairs carry their
// smaller vertex as id (the ids are renumbered by smallest member anyway), and
// the rounds walk a list of the vertices that can still pair.  256^3 hierarchy:
// rounds 41 -> 15 ms, strength graph 9.5 -> 4.6 ms of kernels; 33^3 cubes: 2.3
// ms of kernels and 61 host reads -> 0.7 ms and 4.
#include "hzb_setup.cuh"
#include <algorithm>

namespace hzb {

__device__ __forceinline__ unsigned edge_hash(int i, int j) {
    unsigned lo = (unsigned)min(i, j), hi = (unsigned)max(i, j);
    unsigned x = lo * 0x9e3779b1u ^ (hi + 0x7f4a7c15u + (lo << 6) + (lo >> 2));
    x ^= x >> 16; x *= 0x7feb352du; x ^= x >> 15; x *= 0x846ca68bu; x ^= x >> 16;
    return x;
}

__device__ __forceinline__ bool pm_red(int k, int round) {
    return (hash_u32((unsigned)k * 2654435761u + (unsigned)round * 0x632be5abu) >> 7) & 1u;
}

// edge key: |a_ij| in FP32, then a hash of the unordered pair, then j; whether
// (w, j) beats (bw, best) as seen from k
__device__ __forceinline__ bool pm_better(int k, float w, int j, float bw, int best) {
    if (best < 0 || w > bw) return true;
    if (w != bw) return false;
    const unsigned h = edge_hash(k, j), bh = edge_hash(k, best);
    return h > bh || (h == bh && j > best);
}

constexpr int PM_LEAD = 4, PM_ROUNDS = 96 + PM_LEAD, PM_IDLE = 4;
constexpr int PM_BLOCK = 512;
constexpr int PM_LANES = 8;   // lanes per row of the compaction

// first diagonal entry of every row (0 without one)
__global__ void __launch_bounds__(256)
k_pm_diag(int n, const int *__restrict__ ia, const int *__restrict__ ja,
          const double *__restrict__ a, double *d) {
    const int lane = threadIdx.x % PM_LANES, base = (threadIdx.x & 31) - lane;
    const int groups = gridDim.x * blockDim.x / PM_LANES;
    const int g0 = (blockIdx.x * blockDim.x + threadIdx.x) / PM_LANES;
    const int rows = (n + groups - 1) / groups;   // the warp's lanes stay together
    for (int q = 0; q < rows; ++q) {
        const int i = g0 + q * groups;
        const int b0 = i < n ? ia[i] : 0, b1 = i < n ? ia[i + 1] : 0;
        bool found = false;
        for (int kb = b0;; kb += PM_LANES) {
            const bool more = !found && kb < b1;
            if (!__any_sync(0xffffffffu, more)) break;
            const int k = kb + lane;
            const bool hit = more && k < b1 && ja[k] == i;
            const unsigned m = (__ballot_sync(0xffffffffu, hit) >> base) & ((1u << PM_LANES) - 1u);
            if (more && m) {
                found = true;
                if (lane == __ffs(m) - 1) d[i] = a[k];
            }
        }
        if (i < n && !found && lane == 0) d[i] = 0.0;
    }
}

// The strong entries off the diagonal of row i (construct_strongly_coupled:
// a_ij^2 >= theta^2 |d_i d_j| and a_ij < 0), in order, to cj / cw from
// position ia[i] on; cnt[i] of them.  state[i]: -1 free, -2 isolated (at most
// one strong entry, the diagonal ones counted).
__global__ void __launch_bounds__(256)
k_pm_strong(int n, const int *__restrict__ ia, const int *__restrict__ ja,
            const double *__restrict__ a, const double *__restrict__ d, double th2, int *cj,
            float *cw, int *cnt, int *state, int *ptr) {
    const int lane = threadIdx.x % PM_LANES, base = (threadIdx.x & 31) - lane;
    const unsigned below = (1u << lane) - 1u;
    const int groups = gridDim.x * blockDim.x / PM_LANES;
    const int g0 = (blockIdx.x * blockDim.x + threadIdx.x) / PM_LANES;
    const int rows = (n + groups - 1) / groups;
    for (int q = 0; q < rows; ++q) {
        const int i = g0 + q * groups;
        const int b0 = i < n ? ia[i] : 0, b1 = i < n ? ia[i + 1] : 0;
        const double di = i < n ? d[i] : 0.0;
        int off = 0, self = 0;
        for (int kb = b0; __any_sync(0xffffffffu, kb < b1); kb += PM_LANES) {
            const int k = kb + lane;
            int j = -1;
            double v = 0.0;
            if (k < b1) { j = ja[k]; v = a[k]; }
            const bool dg = j == i && k < b1;
            const bool st = k < b1 && !dg && v < 0e0 && (v * v) >= th2 * fabs(di * d[j]);
            const unsigned m = (__ballot_sync(0xffffffffu, st) >> base) & ((1u << PM_LANES) - 1u);
            const unsigned ms = (__ballot_sync(0xffffffffu, dg) >> base) & ((1u << PM_LANES) - 1u);
            if (st) {
                const int p = b0 + off + __popc(m & below);
                cj[p] = j;
                cw[p] = (float)fabs(v);
            }
            off += __popc(m);
            self += __popc(ms);
        }
        if (i < n && lane == 0) {
            cnt[i] = off;
            state[i] = off + self > 1 ? -1 : -2;
            ptr[i] = -1;
        }
    }
}

// What a vertex sees in its compacted row: the heaviest entry that ok()
// accepts, and whether any neighbour is free.  L lanes share the row, B
// entries of a lane are in flight together (state and ptr gathers come from
// L2).  seen(j): the word ok and free_of judge entry j by.
template <int L, int B, typename Seen, typename Ok, typename Free>
__device__ __forceinline__ void pm_scan(int k, int b0, int b1, const int *__restrict__ cj,
                                        const float *__restrict__ cw, Seen seen, Ok ok,
                                        Free free_of, int *best_out, bool *any_free) {
    const int sub = threadIdx.x % L;
    const unsigned group = L == 32 ? 0xffffffffu : ((1u << L) - 1u) << ((threadIdx.x & 31) - sub);
    int best = -1;
    float bw = -1.0f;
    bool fr = false;
    for (int p0 = b0; p0 < b1; p0 += L * B) {
        int j[B], v[B];
        float w[B];
#pragma unroll
        for (int q = 0; q < B; ++q) {
            const int p = p0 + q * L + sub;
            j[q] = p < b1 ? cj[p] : -1;
            w[q] = p < b1 ? cw[p] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < B; ++q) v[q] = j[q] >= 0 ? seen(j[q]) : 0;
#pragma unroll
        for (int q = 0; q < B; ++q) {
            if (j[q] < 0) continue;
            fr |= free_of(v[q]);
            if (ok(j[q], v[q]) && pm_better(k, w[q], j[q], bw, best)) { best = j[q]; bw = w[q]; }
        }
    }
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) {
        const int j2 = __shfl_xor_sync(group, best, o, L);
        const float w2 = __shfl_xor_sync(group, bw, o, L);
        if (j2 >= 0 && pm_better(k, w2, j2, bw, best)) { best = j2; bw = w2; }
    }
    *best_out = best;
    *any_free = L == 1 ? fr : __any_sync(group, fr);
}

struct PmArrays {
    int n;
    const int *ia, *cnt, *cj;
    const float *cw;
    int *state, *ptr, *lead;
};

// First half of a round, for the m vertices of `from` (null: all): proposals,
// and the next list of the vertices that are free and see a free neighbour
// (the free set only shrinks, so the others cannot pair any more).  In a
// mutual round after the first, a choice that is still free stands.
template <int L, int B>
__device__ __forceinline__ void pm_propose(const PmArrays &A, int round, int m, const int *from,
                                           int *to, int *len) {
    const int lane = threadIdx.x & 31, sub = threadIdx.x % L;
    const int per = (gridDim.x * blockDim.x) / L;
    const bool mutual = round < PM_LEAD;
    const int w0 = (int)((blockIdx.x * blockDim.x + threadIdx.x) & ~31u) / L;   // the warp's first
    for (int t0 = w0; t0 < m; t0 += per) {
        const int t = t0 + lane / L;
        const int k = t < m ? (from ? __ldcg(from + t) : t) : -1;
        bool keep = k >= 0 && __ldcg(A.state + k) == -1;
        if (keep) {
            int best = -1;
            if (mutual && round > 0) {
                best = __ldcg(A.ptr + k);
                if (__ldcg(A.state + best) != -1) best = -1;
            }
            if (best < 0) {
                const int b0 = A.ia[k], b1 = b0 + A.cnt[k];
                const bool red = mutual || pm_red(k, round);
                pm_scan<L, B>(k, b0, b1, A.cj, A.cw,
                              [&](int j) { return round == 0 ? A.state[j] : __ldcg(A.state + j); },
                              [&](int j, int st) {
                                  return red && st == -1 && (mutual || !pm_red(j, round));
                              },
                              [](int st) { return st == -1; }, &best, &keep);
                if (sub == 0) __stcg(A.ptr + k, best);
            }
        }
        const unsigned mask = __ballot_sync(0xffffffffu, keep && sub == 0);
        int base = 0;
        if (lane == 0 && mask) base = atomicAdd(len, __popc(mask));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (keep && sub == 0) __stcg(to + base + __popc(mask & ((1u << lane) - 1u)), k);
    }
}

// Second half: pairs.  Mutual round: the higher end of a mutual choice;
// handshake: a blue vertex and its heaviest proposer.
template <int L, int B>
__device__ __forceinline__ bool pm_accept(const PmArrays &A, int round, int m, const int *from) {
    const int sub = threadIdx.x % L;
    const int per = (gridDim.x * blockDim.x) / L;
    const bool mutual = round < PM_LEAD;
    bool any = false;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) / L; t < m; t += per) {
        const int j = __ldcg(from + t);
        int best = -1;
        if (mutual) {
            const int p = __ldcg(A.ptr + j);
            if (p >= 0 && p < j && __ldcg(A.ptr + p) == j) best = p;
        } else if (!pm_red(j, round)) {
            const int b0 = A.ia[j], b1 = b0 + A.cnt[j];
            bool unused;
            pm_scan<L, B>(j, b0, b1, A.cj, A.cw, [&](int i) { return __ldcg(A.ptr + i); },
                          [&](int, int p) { return p == j; }, [](int) { return false; }, &best,
                          &unused);
        }
        if (best >= 0 && sub == 0) {
            const int id = min(j, best);
            __stcg(A.state + j, id);
            __stcg(A.state + best, id);
            __stcg(A.lead + id, id);
            any = true;
        }
    }
    return any;
}

// All rounds, the leftovers and the numbering.  ctl (zeroed): lengths of the
// rounds' lists (PM_ROUNDS), pairs found flags (PM_ROUNDS), the CTAs' leader
// counts (gridDim.x), then the aggregate count.  state: the pair's id (its
// smaller vertex) once matched; ptr: the proposal (a matched vertex's last one
// points at its partner or nowhere, so nobody free reads it as an offer),
// later a leftover's id; lead[id]: the aggregate's smallest member.  Arrays
// that other SMs write in this launch are read at L2.
// Bound by memory while most vertices are free (round 0 reads every compacted
// row once; a thread per row, enough rows to hide the gathers), then by the
// two barriers of a round and the dependent loads of one row, which 8 lanes
// share once the list is short against the grid: a round over a few thousand
// rows took 35 us with a thread per row and 13 with 8 lanes.
__global__ void __launch_bounds__(PM_BLOCK)
k_pm_match(PmArrays A, int *list0, int *list1, int *agg, int *ctl, unsigned *bar, int *err) {
    __shared__ int sh[32];
    int *len = ctl, *found = ctl + PM_ROUNDS, *sums = ctl + 2 * PM_ROUNDS;
    const int n = A.n;
    const int *ia = A.ia, *cnt = A.cnt, *cj = A.cj;
    int *state = A.state, *ptr = A.ptr, *lead = A.lead;
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, nthr = gridDim.x * blockDim.x;
    unsigned step = 0;
    int m = n;
    const int *from = nullptr;
    for (int round = 0, idle = 0; round < PM_ROUNDS && idle < PM_IDLE; ++round) {
        int *to = round & 1 ? list1 : list0;
        if (m > 4 * nthr) pm_propose<1, 4>(A, round, m, from, to, len + round);
        else pm_propose<8, 2>(A, round, m, from, to, len + round);
        if (!grid_step(bar, ++step * gridDim.x, err)) return;
        m = __ldcg(len + round);
        from = to;
        if (m == 0) break;   // nobody can pair any more
        const bool any = m > 4 * nthr || round < PM_LEAD ? pm_accept<1, 4>(A, round, m, from)
                                                         : pm_accept<8, 2>(A, round, m, from);
        if (__syncthreads_or(any) && threadIdx.x == 0) __stcg(found + round, 1);
        if (!grid_step(bar, ++step * gridDim.x, err)) return;
        idle = round < PM_LEAD || __ldcg(found + round) ? 0 : idle + 1;
    }
    // leftovers: the first aggregated neighbour's id, or one of their own
    for (int k = gtid; k < n; k += nthr) {
        if (__ldcg(state + k) != -1) continue;
        int id = -1;
        const int b0 = ia[k], b1 = b0 + cnt[k];
        for (int p = b0; p < b1 && id < 0; ++p) id = max(id, __ldcg(state + cj[p]));
        if (id < 0) {
            id = k;
            __stcg(lead + k, k);
        } else {
            atomicMin(lead + id, k);
        }
        __stcg(ptr + k, id);
    }
    if (!grid_step(bar, ++step * gridDim.x, err)) return;
    // numbers: the leaders (smallest members) counted in ascending order, a
    // contiguous chunk per CTA
    auto id_of = [&](int v) {
        const int st = __ldcg(state + v);
        return st >= 0 ? st : st == -1 ? __ldcg(ptr + v) : -1;
    };
    const int tiles = (n + PM_BLOCK - 1) / PM_BLOCK;
    const int per = (tiles + gridDim.x - 1) / gridDim.x;
    const int v0 = blockIdx.x * per * PM_BLOCK, v1 = min(n, v0 + per * PM_BLOCK);
    int mine = 0;
    for (int v = v0 + threadIdx.x; v < v1; v += PM_BLOCK) {
        const int id = id_of(v);
        mine += id >= 0 && __ldcg(lead + id) == v;
    }
    int total = 0;
    block_exscan(mine, sh, &total);
    if (threadIdx.x == 0) __stcg(sums + blockIdx.x, total);
    if (!grid_step(bar, ++step * gridDim.x, err)) return;
    int before = 0;
    for (int b = threadIdx.x; b < (int)blockIdx.x; b += PM_BLOCK) before += __ldcg(sums + b);
    block_exscan(before, sh, &before);
    int *number = list0;
    for (int vb = v0; vb < v1; vb += PM_BLOCK) {
        const int v = vb + threadIdx.x;
        const int id = v < v1 ? id_of(v) : -1;
        const bool leader = id >= 0 && __ldcg(lead + id) == v;
        const int ex = block_exscan(leader, sh, &total);
        if (leader) __stcg(number + v, before + ex);
        before += total;
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) sums[gridDim.x] = before;
    if (!grid_step(bar, ++step * gridDim.x, err)) return;
    for (int v = gtid; v < n; v += nthr) {
        const int id = id_of(v);
        agg[v] = id >= 0 ? __ldcg(number + __ldcg(lead + id)) : UNPT;
    }
}

int match_parallel(const DCsr<double> &A, double theta, int *agg, int *nagg, cudaStream_t s) {
    const int n = A.n;
    static int per_sm = 0;   // the same on every device this library runs on
    if (per_sm == 0 &&
        (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pm_match, PM_BLOCK, 0) !=
             cudaSuccess || per_sm < 1))
        per_sm = 1;
    const int grid = std::min(per_sm * sm_count(), div_up(n, PM_BLOCK));
    const int nctl = 2 * PM_ROUNDS + grid + 1;
    double *d = nullptr;
    float *cw = nullptr;
    int *cj = nullptr, *cnt = nullptr, *work = nullptr, *ctl = nullptr;
    int rc = SUCCESS, h[2] = {0, 0};
    cudaError_t e = cudaSuccess;
    if ((rc = dalloc(&d, n)) || (rc = dalloc(&cj, A.nnz)) || (rc = dalloc(&cw, A.nnz)) ||
        (rc = dalloc(&cnt, n)) || (rc = dalloc(&work, (size_t)5 * n)) ||
        (rc = dalloc(&ctl, nctl + 2)))
        goto done;
    {
        int *state = work, *ptr = work + n, *lead = work + (size_t)2 * n;
        int *list0 = work + (size_t)3 * n, *list1 = work + (size_t)4 * n;
        int *err = ctl + nctl;
        unsigned *bar = (unsigned *)(ctl + nctl + 1);
        const int g = grid_for((long long)n * PM_LANES);
        e = cudaMemsetAsync(ctl, 0, sizeof(int) * (nctl + 2), s);
        k_pm_diag<<<g, 256, 0, s>>>(n, A.ia, A.ja, A.val, d);
        k_pm_strong<<<g, 256, 0, s>>>(n, A.ia, A.ja, A.val, d, theta * theta, cj, cw, cnt, state,
                                    ptr);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(PM_BLOCK);
        cfg.stream = s;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (e == cudaSuccess)
            e = cudaLaunchKernelEx(&cfg, k_pm_match,
                                   PmArrays{n, A.ia, cnt, cj, cw, state, ptr, lead}, list0, list1,
                                   agg, ctl, bar, err);
        count_launch(3);
        // the aggregate count and the barrier's error word, side by side
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(h, ctl + nctl - 1, sizeof(h), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    }
    if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; }
    else if (h[1]) {
        set_error_msg("the rounds of the parallel matching ran out of time");
        rc = ERROR_SOLVER_MISC;
    }
    *nagg = h[0];
done:
    dfree(d); dfree(cj); dfree(cw); dfree(cnt); dfree(work); dfree(ctl);
    return rc;
}

}  // namespace hzb
