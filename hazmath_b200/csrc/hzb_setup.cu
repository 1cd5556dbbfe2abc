// hzb_setup.cu -- setup-phase kernels of the UA-AMG hierarchy.
// Compiled with -fmad=false like the cycle kernels: the Galerkin sums are
// rounded in the reference's order.
#include "hzb_setup.cuh"
#include <cooperative_groups.h>
#include <algorithm>
#include <cstdlib>
#include <mutex>
#include <vector>

namespace hzb {

// ---------------------------------------------------------------------------
// exclusive scan (int32)
// ---------------------------------------------------------------------------
constexpr int SCAN_BLOCK = 256, SCAN_ITEMS = 8, SCAN_TILE = SCAN_BLOCK * SCAN_ITEMS;

__global__ void k_scan_tiles(const int *__restrict__ in, int n, int *tiles) {
    __shared__ int sh[32];
    const int base = blockIdx.x * SCAN_TILE;
    int v = 0;
    for (int k = threadIdx.x; k < SCAN_TILE; k += SCAN_BLOCK) {
        int i = base + k;
        if (i < n) v += in[i];
    }
    int tot;
    block_exscan(v, sh, &tot);
    if (threadIdx.x == 0) tiles[blockIdx.x] = tot;
}

__global__ void k_scan_tilesums(int *tiles, int nt) {
    __shared__ int sh[32];
    int carry = 0;
    for (int b = 0; b < nt; b += blockDim.x) {
        int i = b + threadIdx.x;
        int v = i < nt ? tiles[i] : 0;
        int tot;
        int ex = block_exscan(v, sh, &tot);
        if (i < nt) tiles[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) tiles[nt] = carry;
}

__global__ void k_scan_apply(const int *__restrict__ in, int *out, int n,
                             const int *__restrict__ tiles) {
    __shared__ int sh[32];
    const int base = blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int v[SCAN_ITEMS];
    int sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        int i = base + k;
        v[k] = i < n ? in[i] : 0;
        sum += v[k];
    }
    int tot;
    int ex = block_exscan(sum, sh, &tot) + tiles[blockIdx.x];
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; ++k) {
        int i = base + k;
        if (i < n) out[i] = ex;
        ex += v[k];
    }
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = tiles[gridDim.x];
}

int scan_tmp_size(int n) { return div_up(n > 0 ? n : 1, SCAN_TILE) + 1; }

int scan_exclusive(const int *in, int *out, int n, int *tmp, cudaStream_t s) {
    if (n <= 0) {
        HZB_CUDA(cudaMemsetAsync(out, 0, sizeof(int), s));
        return SUCCESS;
    }
    const int nt = div_up(n, SCAN_TILE);
    k_scan_tiles<<<nt, SCAN_BLOCK, 0, s>>>(in, n, tmp);
    k_scan_tilesums<<<1, 1024, 0, s>>>(tmp, nt);
    k_scan_apply<<<nt, SCAN_BLOCK, 0, s>>>(in, out, n, tmp);
    count_launch(3);
    HZB_LAUNCH_CHECK();
    return SUCCESS;
}

// ---------------------------------------------------------------------------
// strength graph
// ---------------------------------------------------------------------------
__global__ void k_first_diag(int n, const int *__restrict__ ia,
                             const int *__restrict__ ja, const double *__restrict__ a,
                             double *d) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        double v = 0.0;
        for (int k = ia[i]; k < ia[i + 1]; ++k)
            if (ja[k] == i) { v = a[k]; break; }
        d[i] = v;
    }
}

__device__ __forceinline__ bool strong(int i, int j, double v, double th2,
                                       const double *d) {
    return j == i || ((v * v) >= th2 * fabs(d[i] * d[j]) && v < 0e0);
}

__global__ void k_strength_count(int n, const int *__restrict__ ia,
                                 const int *__restrict__ ja,
                                 const double *__restrict__ a,
                                 const double *__restrict__ d, double th2,
                                 int *cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        int c = 0;
        for (int k = ia[i]; k < ia[i + 1]; ++k) c += strong(i, ja[k], a[k], th2, d);
        cnt[i] = c;
    }
}

__global__ void k_strength_fill(int n, const int *__restrict__ ia,
                                const int *__restrict__ ja,
                                const double *__restrict__ a,
                                const double *__restrict__ d, double th2,
                                const int *__restrict__ nia, int *nja,
                                double *nval) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        int p = nia[i];
        for (int k = ia[i]; k < ia[i + 1]; ++k)
            if (strong(i, ja[k], a[k], th2, d)) { nja[p] = ja[k]; nval[p] = a[k]; ++p; }
    }
}

int strength_graph(const DCsr<double> &A, double theta, int *nia, int *nja,
                   double *nval, int *nnnz, int *tmp, cudaStream_t s) {
    const int n = A.n;
    double *d = nullptr;
    int *cnt = nullptr;
    HZB_TRY(dalloc(&d, n));
    int rc = dalloc(&cnt, n);
    if (rc) { dfree(d); return rc; }
    const double th2 = theta * theta;
    const int g = grid_for(n);
    k_first_diag<<<g, 256, 0, s>>>(n, A.ia, A.ja, A.val, d);
    k_strength_count<<<g, 256, 0, s>>>(n, A.ia, A.ja, A.val, d, th2, cnt);
    count_launch(2);
    rc = scan_exclusive(cnt, nia, n, tmp, s);
    if (!rc) {
        k_strength_fill<<<g, 256, 0, s>>>(n, A.ia, A.ja, A.val, d, th2, nia, nja, nval);
        count_launch();
        cudaError_t e = cudaMemcpyAsync(nnnz, nia + n, sizeof(int),
                                        cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; }
    }
    dfree(d);
    dfree(cnt);
    return rc;
}

// ---------------------------------------------------------------------------
// heavy edge matching, reference order: one warp walks the vertices in
// ascending order; the 32 lanes examine a row's neighbours together.
// ---------------------------------------------------------------------------
// Candidate order of heavy_edg(w, id, iz-1, 0): the largest weight wins, and
// among equal weights the later position in the row (backward scan, strict >).
__device__ __forceinline__ void better_last(double &w, int &p, double w2, int p2) {
    if (p2 >= 0 && (p < 0 || w2 > w || (w2 == w && p2 > p))) { w = w2; p = p2; }
}
// heavy_edg(w, id, 0, iz-1): largest weight, among equals the earlier position.
__device__ __forceinline__ void better_first(double &w, int &p, double w2, int p2) {
    if (p2 >= 0 && (p < 0 || w2 > w || (w2 == w && p2 < p))) { w = w2; p = p2; }
}

__global__ void __launch_bounds__(32)
k_hem_seq(int n, const int *__restrict__ ia, const int *__restrict__ ja,
          const double *__restrict__ a, int *mask_, int *cnt_, int *out) {
    volatile int *mask = mask_;
    volatile int *cnt = cnt_;
    const int lane = threadIdx.x;
    for (int k = lane; k < n; k += 32) {
        mask[k] = (ia[k + 1] - ia[k] > 1) ? -1 : -2;   // pass 0
        cnt[k] = 0;
    }
    __syncwarp();
    int nc = 0;
    for (int k = 0; k < n; ++k) {                      // pass 1
        if (mask[k] != -1) continue;
        const int b0 = ia[k], b1 = ia[k + 1];
        double bw = 0.0;
        int bp = -1;
        for (int p = b0 + lane; p < b1; p += 32) {
            const int j = ja[p];
            if (j != k && mask[j] < 0) better_last(bw, bp, fabs(a[p]), p);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double w2 = __shfl_xor_sync(0xffffffffu, bw, o);
            int p2 = __shfl_xor_sync(0xffffffffu, bp, o);
            better_last(bw, bp, w2, p2);
        }
        if (bp >= 0) {
            if (lane == 0) {
                const int pick = ja[bp];
                mask[k] = nc;
                mask[pick] = nc;
                cnt[nc] = 2;
            }
            ++nc;
        }
        __syncwarp();
    }
    int status = 0;
    for (int k = 0; k < n; ++k) {                      // pass 2
        if (mask[k] != -1) continue;
        const int b0 = ia[k], b1 = ia[k + 1];
        double bw = 0.0;
        int bp = -1, bc = -1;
        for (int p = b0 + lane; p < b1; p += 32) {
            const int kc = mask[ja[p]];
            if (kc >= 0) {
                double w2 = (double)(-cnt[kc]);
                int oldp = bp;
                better_first(bw, bp, w2, p);
                if (bp != oldp) bc = kc;
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            double w2 = __shfl_xor_sync(0xffffffffu, bw, o);
            int p2 = __shfl_xor_sync(0xffffffffu, bp, o);
            int c2 = __shfl_xor_sync(0xffffffffu, bc, o);
            int oldp = bp;
            better_first(bw, bp, w2, p2);
            if (bp != oldp) bc = c2;
        }
        if (bp < 0) { status = -1; break; }
        if (lane == 0) {
            mask[k] = bc;
            cnt[bc] = cnt[bc] + 1;
        }
        __syncwarp();
    }
    __syncwarp();
    for (int k = lane; k < n; k += 32)                 // pass 3
        if (mask[k] < 0) mask[k] = UNPT;
    if (lane == 0) { out[0] = nc; out[1] = status; }
}

// longest row, for the ranking's limit
__global__ void k_longest_row(int n, const int *__restrict__ ia, int *longest) {
    __shared__ int sh[32];
    int len = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        len = max(len, ia[i + 1] - ia[i]);
    len = block_max(len, sh);
    if (threadIdx.x == 0) atomicMax(longest, len);
}

int longest_row(int n, const int *ia, int *longest, cudaStream_t s) {
    k_longest_row<<<grid_for(n), 256, 0, s>>>(n, ia, longest);
    count_launch();
    HZB_LAUNCH_CHECK();
    return SUCCESS;
}

__global__ void k_hem_init(int n, const int *__restrict__ ia, int *state) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += gridDim.x * blockDim.x)
        state[k] = (ia[k + 1] - ia[k] > 1) ? -1 : -2;   // pass 0
}

// --- pass 1 in rounds over all SMs -------------------------------------------
// Pass 1 of vertex k takes, among the unmatched neighbours j != k, the entry
// of largest |a_kj|, ties to the later position.  That order does not depend
// on the matching state, so a parallel kernel first writes every row's
// neighbours in that order (self entries as -1 at the end).
constexpr int HEM_RANK_MAXLEN = 4096;       // longest row the ranking accepts

// one warp per row: rank of entry p = number of entries that come before it
__global__ void k_hem_rank(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                           const double *__restrict__ a, int *__restrict__ cand) {
    const int lane = threadIdx.x & 31;
    const int nw = (gridDim.x * blockDim.x) >> 5;
    for (int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; k < n; k += nw) {
        const int b0 = ia[k], b1 = ia[k + 1];
        int nself = 0;
        for (int p = b0 + lane; p < b1; p += 32) nself += ja[p] == k;
        for (int o = 16; o > 0; o >>= 1) nself += __shfl_xor_sync(0xffffffffu, nself, o);
        const int nother = b1 - b0 - nself;
        for (int p = b0 + lane; p < b1; p += 32) {
            const int j = ja[p];
            int r = 0;
            if (j != k) {
                const double w = fabs(a[p]);
                for (int q = b0; q < b1; ++q) {
                    if (ja[q] == k) continue;
                    const double w2 = fabs(a[q]);
                    r += (w2 > w) || (w2 == w && q > p);
                }
                cand[b0 + r] = j;
            } else {
                for (int q = b0; q < p; ++q) r += ja[q] == k;
                cand[b0 + nother + r] = -1;
            }
        }
    }
}

// The walk's outcome without the walk.  A row u that is still undecided
// (neither matched nor visited) threatens a vertex v when it might take v at
// its visit: v is u itself, or a free candidate of u not ranked below a
// candidate that is certain to be free for u (one that no undecided row
// before u threatens).  Row u can be decided as soon as no earlier row
// threatens u, and it takes its best free candidate if no earlier row
// threatens that one either: then the walk would find the same state at its
// visit.  Threats only ever shrink, so what held a round ago is a safe bound,
// and one barrier per round is enough: in round r a thread decides its row,
// or posts the row's threats, by the smallest threatening row per vertex that
// round r - 1 posted.  The posts carry the round in their upper half
// (downwards, so a 64-bit minimum prefers the newer round), two arrays in
// turn, and nothing has to be cleared.
//
// The rows in play are a window: a thread that finishes its row takes the
// next one in ascending order, so every row below a row in play is decided or
// in play itself.  A row that has just entered cannot use the previous
// round's posts, which miss the rows that entered with it, and threatens all
// its candidates.  The smallest undecided row is always decided within three
// rounds, so the loop ends.
//
// Bound by the latency of a round (row state, previous posts, barrier: 4 to 5
// us), not by bytes: a walk of one CTA takes 60 to 83 ns per row (167 ms for the
// 2,048,383 rows of the 128^3 log-normal system, 318 ms for its hierarchy; 11.8
// and 30 ms in rounds).
//
// CLUSTER: the CTAs are one cluster of at most 8, whose barrier and counts (in
// every member's shared memory) cost less.  For levels whose rows are all in
// play in it at once, 8192: there it takes 0.88 to 1.0 of the grid's time (2D,
// 3D and anisotropic hierarchies, 2,400 to 8,192 rows; whole call 0.76 against
// 0.69 ms at 4,096 rows of a 2D one).  With more rows its window lengthens the
// dependency chain, and it takes 0.97 to 1.55 (9,600 rows 1.28 against 1.94
// ms, 12,187 0.74 and 0.83, 16,256 1.33 and 2.06, 32,512 1.72 and 4.34).
constexpr int HEM_BLOCK = 1024, HEM_CLUSTER = 8, HEM_CLUSTER_ROWS = HEM_BLOCK * HEM_CLUSTER;

// A chain is decided one row a round.  So every HEM_PACE rounds the rows decided
// in them and the time they took are looked at (the first CTA's, for all; either
// way gives the same map), and the rounds stop for the walk below, which starts
// over, when at this pace, and with it growing on as it did since the window
// before, they would not be through in the walk's time for all rows, hem_walk_ns
// each.  The growth counts: on 2D levels a front builds up for hundreds of rounds,
// and by the pace alone those gave up (500,000 rows: 30 ms instead of 16).  The
// time counts: a round of 4 to 5 us takes 12 to 21 when long rows crowd into a
// narrow band.  Over 150 levels of 2D, anisotropic, 3D and strip hierarchies
// 254 ms (288 in rounds, 651 as walks).  Chains of 100,000 and
// 1,000,000 rows: 281 and 3045 ms in rounds, 6.6 and 61 so; strips of 16 x 7,500
// points 22 and 7.8; 200,000 rows of 30 entries within 300 columns 55 and 19.5.
//   Up to HEM_WALK_SMALL rows the walk goes first: 0.30 to 0.55 ms a call where
// the rounds take 0.34 to 2.2 (2D 0.69 and 0.40, log-normal 3D 0.87 and 0.48,
// constant 3D 0.34 and 0.41, all of about 3,900 rows), and in proportion to the
// rows' length above 25 entries (random graphs of 8,000 rows with 50 entries 2.0
// and 2.2 ms, with 200 3.1 and 8.3; of 16,000 with 100 4.4 and 4.5).
constexpr unsigned HEM_PACE = 32;
constexpr int HEM_WALK_SMALL = 4096, HEM_WALK_ROW = 25;
// the walk takes 60 to 80 ns a row of 5 to 15 entries, 85 to 180 of 30, 220 to 440
// of 100; a third more here, so that it is clearly the faster one
inline float hem_walk_ns(int n, int nnz) { return 85.f + 1.5f * (float)nnz / (float)n; }
// A graph that reaches too far for the walk's ring (524,000 rows) goes on in
// rounds, unless one warp on the rows themselves, 1 us each, is the faster one at
// that (a periodic chain of 600,000 rows: 0.6 s, 1.8 in rounds).
constexpr float HEM_WARP_NS = 1300.f;

template <bool CLUSTER>
__global__ void __launch_bounds__(HEM_BLOCK)
k_hem_rounds(int n, const int *__restrict__ ia, const int *__restrict__ cand, int *state,
             unsigned long long *post, int *next, unsigned long long *bar, int *err,
             float walk_ns, int *stopped, unsigned *window_ns) {
    const int lane = threadIdx.x & 31;
    constexpr int B = 4;             // candidates examined at a time
    __shared__ int s_count[2][HEM_CLUSTER];
    int u = -1, p0 = 0, p1 = 0;      // the row in play, its candidates left
    int pending = blockIdx.x * blockDim.x + threadIdx.x;   // enters next round
    bool more = true;                // rows may be left to take
    GridTally tally;
    unsigned total = 0, paced = 0;   // rows decided, by now and at the last look
    float pace = 0.f;                // in the window before that
    unsigned long long clock = 0;    // of the first CTA's first thread
    const unsigned max_round = 3u * (unsigned)n + 16u;
    for (unsigned r = 1;; ++r) {
        const unsigned long long *prev = post + (size_t)((r - 1) & 1u) * n;
        unsigned long long *cur = post + (size_t)(r & 1u) * n;
        const unsigned long long mark = (unsigned long long)(0xffffffffu - r) << 32;
        const unsigned was = 0xffffffffu - (r - 1);
        const bool fresh = u < 0;
        bool done = false;           // its row is decided in this round
        if (u < 0 && pending < n) {
            u = pending;
            p0 = ia[u];
            p1 = ia[u + 1];
        }
        if (u >= 0) {
            // smallest row that threatened v in the previous round
            auto threat = [&](unsigned long long t) {
                return (unsigned)(t >> 32) == was ? (int)(unsigned)t : 0x7fffffff;
            };
            const int su = __ldcg(state + u);
            const unsigned long long tu = __ldcg(prev + u);
            done = su != -1;                       // an earlier row took it
            const bool mine = !fresh && threat(tu) == u;
            int best = -1;
            bool open = true;
            for (int p = p0; open && p < p1; p += B) {
                int c[B], sc[B];
                unsigned long long t[B];
#pragma unroll
                for (int q = 0; q < B; ++q) c[q] = p + q < p1 ? cand[p + q] : -1;
#pragma unroll
                for (int q = 0; q < B; ++q) {
                    sc[q] = c[q] >= 0 ? __ldcg(state + c[q]) : 0;
                    t[q] = c[q] >= 0 ? __ldcg(prev + c[q]) : 0ull;
                }
                if (done) break;
#pragma unroll
                for (int q = 0; q < B; ++q) {
                    if (!open) continue;
                    if (c[q] < 0) { open = false; continue; }   // end of the list
                    if (sc[q] >= 0) continue;                   // matched
                    const int tv = threat(t[q]);
                    if (best < 0) {
                        best = c[q];
                        p0 = p + q;           // what precedes it stays matched
                        if (mine && tv == u) {
                            __stcg(state + u, u);
                            __stcg(state + best, u);
                            done = true;
                            open = false;
                            continue;
                        }
                    }
                    atomicMin(cur + c[q], mark | (unsigned)u);
                    if (!fresh && tv >= u) open = false;        // free for u for certain
                }
            }
            if (best < 0 && mine) done = true;   // visited without a partner
            if (!done) atomicMin(cur + u, mark | (unsigned)u);
            if (done) u = -1;
        }
        if (walk_ns > 0.f && r % HEM_PACE == 0 && blockIdx.x == 0 && threadIdx.x == 0) {
            unsigned long long now;
            asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
            __stcg(window_ns, (unsigned)min(now - clock, 0xffffffffull));
            clock = now;
        }
        // rows for the threads without one, ascending
        const unsigned need = __ballot_sync(0xffffffffu, u < 0);
        int base = n;
        const int lead = __ffs(need) - 1;
        if (more && lane == lead) base = atomicAdd(next, __popc(need));
        if (CLUSTER) {
            namespace cg = cooperative_groups;
            cg::cluster_group cl = cg::this_cluster();
            const int count = __syncthreads_count(done);
            if (threadIdx.x < gridDim.x)
                *cl.map_shared_rank(&s_count[r & 1u][blockIdx.x], threadIdx.x) = count;
            cl.sync();
            for (unsigned q = 0; q < gridDim.x; ++q) total += (unsigned)s_count[r & 1u][q];
        } else if (!grid_tally(bar, tally, done, &total, err)) {
            return;
        }
        if (total == (unsigned)n) return;
        if (walk_ns > 0.f && r % HEM_PACE == 0) {
            // the same for every CTA: only the common count and time go in
            const float d = (float)(total - paced);
            const float w = (float)n * walk_ns / fmaxf(1.f, (float)__ldcg(window_ns));
            if (r > HEM_PACE &&
                d * w + 0.5f * fmaxf(0.f, d - pace) * w * w < (float)(n - (int)total)) {
                if (blockIdx.x == 0 && threadIdx.x == 0) *stopped = 1;
                return;
            }
            pace = d;
            paced = total;
        }
        if (need) {
            base = __shfl_sync(0xffffffffu, base, lead);
            pending = n;
            if (u < 0) pending = min(n, base + __popc(need & ((1u << lane) - 1u)));
            if (base >= n) more = false;
        }
        if (r >= max_round) {
            if (blockIdx.x == 0 && threadIdx.x == 0) *err = 1;
            return;
        }
    }
}

// --- pass 1 as a walk ---------------------------------------------------------
// For graphs whose rows can only be decided one after the other (a chain, a
// narrow strip), where the rounds above give up: one CTA streams the ranked
// lists through shared memory in tiles of 32 rows with cp.async, HEM_PIPE tiles
// ahead of the tile it works on, so no global load latency sits on its critical
// path (83 ns a row), and only looks for the first unmatched entry of a list.
constexpr int HEM_RING_BITS = 1 << 20;                 // 128 KB of shared memory
constexpr int HEM_RING_WORDS = HEM_RING_BITS / 32;
constexpr int HEM_PIPE = 4;                 // tiles in flight ahead of the walk
constexpr int HEM_TILE_CAP = 3072;          // staged candidates per tile
// slots: the tiles in flight plus the one being walked
constexpr int HEM_IA_SLOTS = 2 * HEM_PIPE + 2, HEM_IA_STRIDE = 36;
constexpr int HEM_C_SLOTS = HEM_PIPE + 2;
constexpr int HEM_MISC_WORDS = 32 * 2 + 32 + 2 * 32 + 2;   // info, Pm, picks, accepted
constexpr size_t HEM_STAGED_SMEM =
    (size_t)HEM_RING_WORDS * 4 + (size_t)HEM_C_SLOTS * HEM_TILE_CAP * 4 +
    (size_t)HEM_IA_SLOTS * HEM_IA_STRIDE * 4 + (size_t)HEM_MISC_WORDS * 4;

__global__ void k_graph_bandwidth(int n, const int *__restrict__ ia,
                                  const int *__restrict__ ja, int *bw) {
    __shared__ int sh[32];
    int b = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        for (int k = ia[i]; k < ia[i + 1]; ++k) b = max(b, abs(ja[k] - i));
    b = block_max(b, sh);
    if (threadIdx.x == 0) atomicMax(bw, b);
}

__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// The matched state of the vertices in play lives in a ring of shared memory:
// one byte per vertex (BYTES, 2^17 vertices, plain stores) while the window
// fits, else one bit per vertex (2^20 vertices, atomicOr).  Both rings take
// 128 KB.  Ring size > 2 bw + 64: the 32 slots entering the window are
// cleared when a tile begins (vertices >= r0 + bw cannot be matched before
// tile r0 starts, and the slot's previous owner lies below r0 - bw).
template <bool BYTES>
struct HemRing {
    static constexpr unsigned SIZE = BYTES ? (1u << 17) : (1u << 20);
    static constexpr unsigned RM = SIZE - 1;
    void *mem;
    __device__ __forceinline__ bool get(int v) const {
        const unsigned u = (unsigned)v & RM;
        if (BYTES) return ((const volatile unsigned char *)mem)[u] != 0;
        return (((const volatile unsigned *)mem)[u >> 5] >> (u & 31)) & 1u;
    }
    __device__ __forceinline__ void set(int v) {
        const unsigned u = (unsigned)v & RM;
        if (BYTES) ((volatile unsigned char *)mem)[u] = 1;
        else atomicOr((unsigned *)mem + (u >> 5), 1u << (u & 31));
    }
    // vertices v0 .. v0 + 31, by the whole warp
    __device__ __forceinline__ void clear32(int v0, int lane) {
        if (BYTES) {
            ((unsigned char *)mem)[((unsigned)v0 + lane) & RM] = 0;
        } else {
            const unsigned u = (unsigned)v0 & RM, sh = u & 31u, w0 = u >> 5;
            unsigned *w = (unsigned *)mem;
            if (lane == 0) w[w0] &= ~(0xffffffffu << sh);
            if (lane == 1 && sh) w[(w0 + 1) & (SIZE / 32 - 1)] &= ~((1u << sh) - 1u);
        }
    }
};

// Two warps.  Warp 1 streams row pointers and ranked lists into shared
// memory (cp.async, HEM_PIPE tiles ahead) and writes the pairs of finished
// tiles to mask/cnt; warp 0 walks the tiles.  Within a tile of 32 rows every
// row first takes its best candidate unmatched when the tile starts; rows are
// then settled in order.  A row keeps that choice unless an earlier row of
// the tile took it or matched the row's choice (vertices only ever become
// matched, so the entries ranked above it stay ineligible); such a row scans
// its list again.  For a row that keeps its choice the effect on the rows
// after it is known in advance: the row it picks leaves the walk (rm) and the
// rows that wanted the same vertex or this row go stale (st).
template <bool BYTES>
__global__ void __launch_bounds__(64)
k_hem_pass1_staged(int n, int bw, const int *__restrict__ ia, const int *__restrict__ cand,
                   int *mask, int *cnt, int *out) {
    extern __shared__ unsigned hem_smem[];
    HemRing<BYTES> ring{hem_smem};
    int *cbuf = (int *)(hem_smem + HEM_RING_WORDS);
    int *iabuf = cbuf + HEM_C_SLOTS * HEM_TILE_CAP;
    uint2 *info = (uint2 *)(iabuf + HEM_IA_SLOTS * HEM_IA_STRIDE);
    unsigned *pm = (unsigned *)(info + 32);
    int *picks = (int *)(pm + 32);              // [2][32], by tile parity
    unsigned *accepted = (unsigned *)(picks + 64);   // [2]
    const int lane = threadIdx.x & 31;
    const int ntiles = (n + 31) >> 5;

    if (threadIdx.x >= 32) {   // ---- warp 1: staging and output
        int nc = 0;
        auto emit = [&](int u) {
            const unsigned acc = accepted[u & 1];
            if ((acc >> lane) & 1u) {
                const int id = nc + __popc(acc & ((1u << lane) - 1u));
                const int q = picks[(u & 1) * 32 + lane];
                mask[(u << 5) + lane] = id;
                mask[q] = id;
                cnt[id] = 2;
            }
            nc += __popc(acc);
        };
        for (int j = -2 * HEM_PIPE; j < ntiles; ++j) {
            if (j >= 2) emit(j - 2);
            const int ui = j + 2 * HEM_PIPE;   // row pointers of tile j + 2 PIPE
            if (ui < ntiles) {
                const int r0 = ui << 5, rows = min(32, n - r0);
                int *dst = iabuf + (ui % HEM_IA_SLOTS) * HEM_IA_STRIDE;
                cp_async4(dst + lane, ia + r0 + min(lane, rows));
                if (lane == 0) cp_async4(dst + 32, ia + r0 + rows);
            }
            cp_async_wait<HEM_PIPE - 1>();   // ia(j + PIPE) and cand(j) have landed
            __syncwarp();
            const int uc = j + HEM_PIPE;     // ranked lists of tile j + PIPE
            if (uc >= 0 && uc < ntiles) {
                const int *iu = iabuf + (uc % HEM_IA_SLOTS) * HEM_IA_STRIDE;
                const int rows = min(32, n - (uc << 5));
                const int e0 = iu[0], m = iu[rows] - e0;
                if (m <= HEM_TILE_CAP) {
                    int *dst = cbuf + (uc % HEM_C_SLOTS) * HEM_TILE_CAP;
                    for (int e = lane; e < m; e += 32) cp_async4(dst + e, cand + e0 + e);
                }
            }
            cp_async_commit();
            if (j >= 0) __syncthreads();   // tile j is ready; tile j - 1 is walked
        }
        cp_async_wait<0>();
        __syncthreads();                    // the last tile is walked
        if (ntiles >= 2) emit(ntiles - 2);
        if (ntiles >= 1) emit(ntiles - 1);
        if (lane == 0) out[0] = nc;
        return;
    }

    // ---- warp 0: the walk
    for (int w = lane; w < HEM_RING_WORDS; w += 32) hem_smem[w] = 0u;
    __syncthreads();
    for (int t = 0; t < ntiles; ++t) {
        const int r0 = t << 5, rows = min(32, n - r0);
        ring.clear32(r0 + bw, lane);
        __syncwarp();
        const int *it = iabuf + (t % HEM_IA_SLOTS) * HEM_IA_STRIDE;
        const int e0 = it[0];
        const bool staged = it[rows] - e0 <= HEM_TILE_CAP;
        const int *ct = staged ? cbuf + (t % HEM_C_SLOTS) * HEM_TILE_CAP : cand;
        const int off = staged ? e0 : 0;
        int *pk = picks + (t & 1) * 32;
        // rows of the tile still unmatched and not isolated (pass 0)
        const bool act = lane < rows && it[lane + 1] - it[lane] > 1 && !ring.get(r0 + lane);
        unsigned todo = __ballot_sync(0xffffffffu, act);
        int p = -1;
        if (act) {
            const int b1 = it[lane + 1];
            for (int e = it[lane]; e < b1; e += 2) {
                const int c0 = ct[e - off];
                const int c1 = e + 1 < b1 ? ct[e + 1 - off] : -1;
                const bool ok0 = c0 >= 0 && !ring.get(c0);
                const bool ok1 = c1 >= 0 && !ring.get(c1);
                if (ok0) { p = c0; break; }
                if (ok1) { p = c1; break; }
            }
        }
        const unsigned tl = (unsigned)(p - r0);   // < 32: the pick is a row of this tile
        pm[lane] = 0u;
        __syncwarp();
        if (p >= 0 && tl < 32u) atomicOr(pm + tl, 1u << lane);
        const unsigned same = __match_any_sync(0xffffffffu, p);
        const unsigned has = __ballot_sync(0xffffffffu, p >= 0);
        __syncwarp();
        if (p >= 0) info[lane] = make_uint2(tl < 32u ? 1u << tl : 0u, same | pm[lane]);
        else info[lane] = make_uint2(0u, 0u);
        pk[lane] = p;
        __syncwarp();
        unsigned stale = 0u, done = 0u, racc = 0u, written = 0u;
        while (todo) {
            const int i = __ffs(todo) - 1;
            todo &= todo - 1u;
            if ((stale >> i) & 1u) {
                // the ring takes every pick of the tile so far, then row i scans again
                const unsigned w = done & has & ~written;
                if ((w >> lane) & 1u) { ring.set(r0 + lane); ring.set(p); }
                written |= w;
                __syncwarp();
                const int b0 = it[i], b1 = it[i + 1];
                int q = -1;
                for (int e = b0; e < b1; e += 32) {
                    const int c = e + lane < b1 ? ct[e + lane - off] : -1;
                    const bool ok = c >= 0 && !ring.get(c);
                    const unsigned bal = __ballot_sync(0xffffffffu, ok);
                    if (bal) {
                        q = __shfl_sync(0xffffffffu, c, __ffs(bal) - 1);
                        break;
                    }
                }
                if (q >= 0) {
                    if (lane == 0) { ring.set(r0 + i); ring.set(q); pk[i] = q; }
                    racc |= 1u << i;
                    const unsigned d = (unsigned)(q - r0);
                    if (d < 32u) todo &= ~(1u << d);
                    stale |= __ballot_sync(0xffffffffu, p == q || p == r0 + i);
                }
                __syncwarp();
                continue;
            }
            const uint2 f = info[i];
            done |= 1u << i;
            todo &= ~f.x;
            stale |= f.y;
        }
        const unsigned acc = (done & has) | racc;
        const unsigned w = done & has & ~written;
        if ((w >> lane) & 1u) { ring.set(r0 + lane); ring.set(p); }
        if (lane == 0) accepted[t & 1] = acc;
        __syncthreads();   // tile t walked; tile t + 1 staged
    }
}

// pairs numbered by their visiting row (state[k] == k), as the walk counts
__global__ void k_hem_visitors(int n, const int *__restrict__ state, int *flag) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x)
        flag[k] = state[k] == k;
}
// state (visiting rows) -> aggregate ids, and the members counted for pass 2
__global__ void k_hem_number(int n, const int *__restrict__ pos, int *state, int *cnt) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n; k += gridDim.x * blockDim.x) {
        const int v = state[k];
        if (v >= 0) {
            state[k] = pos[v];
            if (v == k) cnt[pos[v]] = 2;
        }
    }
}

__global__ void k_flag_eq(int n, const int *__restrict__ v, int val, int *flag) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        flag[i] = v[i] == val;
}
__global__ void k_compact(int n, const int *__restrict__ flag, const int *__restrict__ pos,
                          int *list) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        if (flag[i]) list[pos[i]] = i;
}

// Pass 2 over the leftover list (ascending), one warp: a leftover joins the
// adjacent aggregate with the fewest members, the first such entry on ties,
// and the next leftover sees that aggregate one larger.  A lane takes one
// leftover each and chooses as if no other lane did; the choice stands unless
// an earlier lane chose an aggregate that this row looks at, or is itself a
// neighbour of this row.  Those are looked up by hash in two shared tables of
// the first lane per slot (a false hit only ends the batch early), the lanes
// before the first doubtful one commit, and the next batch starts there.  One
// row at a time took 1.06 ms for the leftovers of the 128^3 log-normal level,
// a chain of four dependent loads each.
__global__ void __launch_bounds__(32)
k_hem_pass2_list(int m, const int *__restrict__ list, const int *__restrict__ ia,
                 const int *__restrict__ ja, int *mask_, int *cnt_, int *out) {
    constexpr int H = 1024;
    __shared__ int lane_of_agg[H], lane_of_row[H];
    volatile int *mask = mask_;
    volatile int *cnt = cnt_;
    const int lane = threadIdx.x;
    for (int q = lane; q < H; q += 32) lane_of_agg[q] = lane_of_row[q] = 32;
    __syncwarp();
    int status = 0;
    for (int q0 = 0; q0 < m;) {
        const int q = q0 + lane;
        const bool on = q < m;
        const int k = on ? list[q] : 0;
        const int b0 = on ? ia[k] : 0, b1 = on ? ia[k + 1] : 0;
        int bc = -1, bn = 0;
        for (int p = b0; p < b1; ++p) {
            const int kc = mask[ja[p]];
            if (kc < 0) continue;
            const int c = cnt[kc];
            if (bc < 0 || c < bn) { bc = kc; bn = c; }
        }
        if (on) {
            if (bc >= 0) atomicMin(lane_of_agg + (bc & (H - 1)), lane);
            atomicMin(lane_of_row + (k & (H - 1)), lane);
        }
        __syncwarp();
        bool doubt = false;
        for (int p = b0; p < b1; ++p) {
            const int j = ja[p], kc = mask[j];
            doubt |= lane_of_row[j & (H - 1)] < lane;
            if (kc >= 0) doubt |= lane_of_agg[kc & (H - 1)] < lane;
        }
        const unsigned dm = __ballot_sync(0xffffffffu, doubt);
        const int stop = dm ? __ffs(dm) - 1 : min(32, m - q0);   // lane 0 has no doubt
        // a row without an aggregated neighbour: the reference stops there
        const unsigned none = __ballot_sync(0xffffffffu, on && lane < stop && bc < 0);
        const int last = none ? __ffs(none) - 1 : stop;
        if (on && bc >= 0) lane_of_agg[bc & (H - 1)] = 32;
        if (on) lane_of_row[k & (H - 1)] = 32;
        if (on && lane < last) {
            mask[k] = bc;
            cnt[bc] = bn + 1;   // no other lane below last chose bc
        }
        __threadfence_block();
        __syncwarp();
        if (none) { status = -1; break; }
        q0 += stop;
    }
    if (lane == 0) out[1] = status;
}

__global__ void k_hem_final(int n, int *mask) {
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < n;
         k += gridDim.x * blockDim.x)
        if (mask[k] < 0) mask[k] = UNPT;
}

int hem_exact(int n, const int *nia, const int *nja, const double *nval,
              int *agg, int *nagg, int *work_n, cudaStream_t s) {
    // out: aggregates, status | longest row | next row | barrier (4) | error, stopped,
    // a window's time
    enum { O_NC = 0, O_STATUS = 1, O_LEN = 2, O_NEXT = 3, O_BAR = 4, O_ERR = 8, O_STOP = 9,
           O_NS = 10, O_N = 12 };
    int *out = nullptr;
    HZB_TRY(dalloc(&out, O_N));
    int h[O_N] = {0};
    int gnnz = 0, rc = SUCCESS;
    const int g = grid_for(n);
    cudaError_t e = cudaMemsetAsync(out, 0, O_N * sizeof(int), s);
    k_longest_row<<<g, 256, 0, s>>>(n, nia, out + O_LEN);
    count_launch();
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(h, out, O_N * sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&gnnz, nia + n, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { dfree(out); set_error(e, __FILE__, __LINE__); return ERROR_SOLVER_MISC; }
    // Rounds over ranked lists, and the walk over them where the rounds' pace is
    // too slow; a warp on the rows themselves for rows longer than the ranking
    // takes (its work grows with the square of a row's length).  HZB_HEM_PATH
    // names one for tests: 1 the rounds to their end, 2 the walk, 4 the warp.
    int path = h[O_LEN] <= HEM_RANK_MAXLEN ? 0 : 4;
    if (const char *f = getenv("HZB_HEM_PATH")) {
        const int want = atoi(f);
        if (want == 4 || (path == 0 && (want == 1 || want == 2))) path = want;
    }
    if (path == 0 &&
        n <= (long long)HEM_WALK_SMALL * std::max<long long>(HEM_WALK_ROW, gnnz / n) / HEM_WALK_ROW)
        path = 2;
    if (path != 4) {
        int *cand = nullptr, *flag = nullptr, *pos = nullptr, *tmp = nullptr, m = 0;
        unsigned long long *post = nullptr;
        int *cnt = work_n;
        if ((rc = dalloc(&cand, gnnz)) || (rc = dalloc(&post, (size_t)2 * n)) ||
            (rc = dalloc(&flag, n)) || (rc = dalloc(&pos, n + 1)) ||
            (rc = dalloc(&tmp, scan_tmp_size(n + 1)))) {
            dfree(cand); dfree(post); dfree(flag); dfree(pos); dfree(tmp); dfree(out);
            return rc;
        }
        auto rank = [&]() {
            k_hem_init<<<g, 256, 0, s>>>(n, nia, agg);
            k_hem_rank<<<std::min(div_up(n, 8), 148 * 64), 256, 0, s>>>(n, nia, nja, nval, cand);
            count_launch(2);
        };
        // the rows left over by pass 1, ascending, and how many (with out)
        auto leftovers = [&]() -> int {
            k_flag_eq<<<g, 256, 0, s>>>(n, agg, -1, flag);
            HZB_TRY(scan_exclusive(flag, pos, n, tmp, s));
            // the ranked lists are done with (gnnz >= leftovers)
            k_compact<<<g, 256, 0, s>>>(n, flag, pos, cand);
            count_launch(2);
            HZB_CUDA(cudaMemcpyAsync(&m, pos + n, sizeof(int), cudaMemcpyDeviceToHost, s));
            HZB_CUDA(cudaMemcpyAsync(h, out, O_N * sizeof(int), cudaMemcpyDeviceToHost, s));
            HZB_CUDA(cudaStreamSynchronize(s));
            return SUCCESS;
        };
        auto rounds = [&](float walk_ns) -> int {
            rank();
            // all ones: older than any round's post
            HZB_CUDA(cudaMemsetAsync(post, 0xff, sizeof(unsigned long long) * 2 * n, s));
            // one CTA per SM; a cluster of 1 to 8 on small levels
            const bool cluster = n <= HEM_CLUSTER_ROWS;
            int grid = std::min(sm_count(), div_up(n, HEM_BLOCK));
            if (cluster) {
                const int want = std::min(grid, HEM_CLUSTER);
                for (grid = 1; grid < want;) grid *= 2;
            }
            const int first = grid * HEM_BLOCK;
            HZB_CUDA(cudaMemsetAsync(out + O_BAR, 0, sizeof(int) * (O_N - O_BAR), s));
            HZB_CUDA(cudaMemcpyAsync(out + O_NEXT, &first, sizeof(int), cudaMemcpyHostToDevice,
                                     s));
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(grid);
            cfg.blockDim = dim3(HEM_BLOCK);
            cfg.stream = s;
            cudaLaunchAttribute attr[1];
            if (cluster) {
                attr[0].id = cudaLaunchAttributeClusterDimension;
                attr[0].val.clusterDim.x = grid;
                attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            } else {
                attr[0].id = cudaLaunchAttributeCooperative;
                attr[0].val.cooperative = 1;
            }
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            HZB_CUDA(cudaLaunchKernelEx(
                &cfg, cluster ? k_hem_rounds<true> : k_hem_rounds<false>, n, nia,
                (const int *)cand, agg, post, out + O_NEXT, (unsigned long long *)(out + O_BAR),
                out + O_ERR, walk_ns, out + O_STOP, (unsigned *)(out + O_NS)));
            k_hem_visitors<<<g, 256, 0, s>>>(n, agg, flag);
            count_launch(2);
            HZB_TRY(scan_exclusive(flag, pos, n, tmp, s));
            k_hem_number<<<g, 256, 0, s>>>(n, pos, agg, cnt);
            count_launch();
            HZB_CUDA(cudaMemcpyAsync(out + O_NC, pos + n, sizeof(int), cudaMemcpyDeviceToDevice,
                                     s));
            return leftovers();
        };
        // *done: false when the graph reaches too far for the walk's ring
        auto walk = [&](bool *done) -> int {
            int bw = n - 1;
            if (bw >= ((int)HemRing<true>::SIZE - 64) / 2) {
                HZB_CUDA(cudaMemsetAsync(out + O_LEN, 0, sizeof(int), s));
                k_graph_bandwidth<<<g, 256, 0, s>>>(n, nia, nja, out + O_LEN);
                count_launch();
                HZB_CUDA(cudaMemcpyAsync(&bw, out + O_LEN, sizeof(int), cudaMemcpyDeviceToHost,
                                         s));
                HZB_CUDA(cudaStreamSynchronize(s));
            }
            *done = bw < (HEM_RING_BITS - 64) / 2;
            if (!*done) return SUCCESS;
            rank();
            auto kernel = bw < ((int)HemRing<true>::SIZE - 64) / 2 ? k_hem_pass1_staged<true>
                                                                   : k_hem_pass1_staged<false>;
            HZB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)HEM_STAGED_SMEM));
            kernel<<<1, 64, HEM_STAGED_SMEM, s>>>(n, bw, nia, cand, agg, cnt, out);
            count_launch();
            return leftovers();
        };
        bool walked = false;
        if (path != 2) rc = rounds(path == 0 ? hem_walk_ns(n, gnnz) : 0.f);
        if (!rc && (path == 2 || h[O_STOP])) {
            rc = walk(&walked);
            if (!rc && !walked) rc = rounds(HEM_WARP_NS);
            if (!rc && !walked && h[O_STOP]) path = 4;
        }
        if (!rc && !h[O_ERR] && path != 4) {
            if (m > 0) {
                k_hem_pass2_list<<<1, 32, 0, s>>>(m, cand, nia, nja, agg, cnt, out);
                count_launch();
            }
            k_hem_final<<<g, 256, 0, s>>>(n, agg);
            count_launch();
        }
        dfree(cand); dfree(post); dfree(flag); dfree(pos); dfree(tmp);
    }
    if (!rc && path == 4) {   // the whole state in global memory
        k_hem_seq<<<1, 32, 0, s>>>(n, nia, nja, nval, agg, work_n, out);
        count_launch();
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, out, O_N * sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    dfree(out);
    if (rc) return rc;
    if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); return ERROR_SOLVER_MISC; }
    if (h[O_ERR]) {
        set_error_msg("the rounds of the heavy edge matching ran out of time");
        return ERROR_SOLVER_MISC;
    }
    *nagg = h[O_NC];
    return h[O_STATUS] < 0 ? ERROR_AMG_COARSEING : SUCCESS;
}

// ---------------------------------------------------------------------------
// Caller-supplied Galerkin inputs, checked before any kernel indexes by them
// (read-only): aggregate ids in [-1, nc), row pointers non-decreasing from 0
// to nnz, column indices in [0, n).  Bits of *bad: 1 aggregate id, 2 row
// pointers, 4 column index.
// ---------------------------------------------------------------------------
__global__ void k_check_rap_inputs(int n, int nnz, const int *__restrict__ ia,
                                   const int *__restrict__ ja, int nc,
                                   const int *__restrict__ agg, int *bad) {
    int b = 0;
    const int m = n > nnz ? n : nnz;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m;
         i += gridDim.x * blockDim.x) {
        if (i < n) {
            const int c = agg[i];
            if (c < -1 || c >= nc) b |= 1;
            if (ia[i + 1] < ia[i]) b |= 2;
        }
        if (i < nnz) {
            const int j = ja[i];
            if (j < 0 || j >= n) b |= 4;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && (ia[0] != 0 || ia[n] != nnz)) b |= 2;
    if (b) atomicOr(bad, b);
}

int check_rap_inputs(int n, int nnz, const int *ia, const int *ja, int nc, const int *agg,
                     int *d_bad, cudaStream_t s) {
    HZB_CUDA(cudaMemsetAsync(d_bad, 0, sizeof(int), s));
    k_check_rap_inputs<<<grid_for(n > nnz ? n : nnz), 256, 0, s>>>(n, nnz, ia, ja, nc, agg,
                                                                    d_bad);
    count_launch();
    int bad = 0;
    HZB_CUDA(cudaMemcpyAsync(&bad, d_bad, sizeof(int), cudaMemcpyDeviceToHost, s));
    HZB_CUDA(cudaStreamSynchronize(s));
    if (bad & 1) {
        set_error_msg("Galerkin product: an aggregate id lies outside [-1, nc)");
        return ERROR_INPUT_PAR;
    }
    if (bad & 2) {
        set_error_msg("Galerkin product: row pointers do not rise from 0 to nnz");
        return ERROR_INPUT_PAR;
    }
    if (bad & 4) {
        set_error_msg("Galerkin product: a column index lies outside [0, n)");
        return ERROR_INPUT_PAR;
    }
    return SUCCESS;
}

// ---------------------------------------------------------------------------
// R = P^T pattern with ascending fine indices per row
// ---------------------------------------------------------------------------
__global__ void k_agg_count(int n, const int *__restrict__ agg, int *cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        if (agg[i] >= 0) atomicAdd(cnt + agg[i], 1);
}
__global__ void k_agg_fill(int n, const int *__restrict__ agg,
                           const int *__restrict__ ria, int *fillc, int *rja) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        const int c = agg[i];
        if (c >= 0) rja[ria[c] + atomicAdd(fillc + c, 1)] = i;
    }
}
__global__ void k_sort_rows(int nr, const int *__restrict__ ia, int *ja) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nr;
         r += gridDim.x * blockDim.x) {
        const int b0 = ia[r], b1 = ia[r + 1];
        for (int p = b0 + 1; p < b1; ++p) {      // insertion sort (short rows)
            int v = ja[p], q = p - 1;
            while (q >= b0 && ja[q] > v) { ja[q + 1] = ja[q]; --q; }
            ja[q + 1] = v;
        }
    }
}

int restriction_pattern(int n, int nc, const int *agg, int *ria, int *rja,
                        int *tmp, cudaStream_t s) {
    int *cnt = nullptr;
    HZB_TRY(dalloc(&cnt, nc));
    HZB_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * (nc > 0 ? nc : 1), s));
    k_agg_count<<<grid_for(n), 256, 0, s>>>(n, agg, cnt);
    count_launch();
    int rc = scan_exclusive(cnt, ria, nc, tmp, s);
    if (!rc) {
        cudaMemsetAsync(cnt, 0, sizeof(int) * (nc > 0 ? nc : 1), s);
        k_agg_fill<<<grid_for(n), 256, 0, s>>>(n, agg, ria, cnt, rja);
        k_sort_rows<<<grid_for(nc), 256, 0, s>>>(nc, ria, rja);
        count_launch(2);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; }
    }
    dfree(cnt);
    return rc;
}

// ---------------------------------------------------------------------------
// Galerkin product A_c = R A P for unit aggregation P (exact order)
// ---------------------------------------------------------------------------
__global__ void k_rap_bound(int nc, const int *__restrict__ ria,
                            const int *__restrict__ rja, const int *__restrict__ ia,
                            int *ub) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc;
         c += gridDim.x * blockDim.x) {
        int u = 1;
        for (int q = ria[c]; q < ria[c + 1]; ++q) {
            const int i = rja[q];
            u += ia[i + 1] - ia[i];
        }
        ub[c] = u;
    }
}

// One thread per coarse row builds its slot list in scratch: slot 0 is the
// diagonal (0.0, accumulated); other columns in first-encounter order; a new
// column takes the entry's value, a known column adds it.
__global__ void k_rap_build(int nc, const int *__restrict__ ria,
                            const int *__restrict__ rja, const int *__restrict__ ia,
                            const int *__restrict__ ja, const double *__restrict__ a,
                            const int *__restrict__ agg, const int *__restrict__ off,
                            int *scol, double *sval, int *rowcnt) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc;
         c += gridDim.x * blockDim.x) {
        int *cols = scol + off[c];
        double *vals = sval + off[c];
        int cnt = 1;
        cols[0] = c;
        vals[0] = 0.0;
        for (int q = ria[c]; q < ria[c + 1]; ++q) {
            const int i = rja[q];
            for (int k = ia[i]; k < ia[i + 1]; ++k) {
                const int cc = agg[ja[k]];
                if (cc < 0) continue;
                int pos = -1;
                for (int t = 0; t < cnt; ++t)
                    if (cols[t] == cc) { pos = t; break; }
                if (pos >= 0) {
                    vals[pos] += a[k];
                } else {
                    cols[cnt] = cc;
                    vals[cnt] = a[k];
                    ++cnt;
                }
            }
        }
        rowcnt[c] = cnt;
    }
}

// slot lists in scratch to CSR
__global__ void k_rap_compact(int nc, const int *__restrict__ off,
                              const int *__restrict__ cia,
                              const int *__restrict__ scol,
                              const double *__restrict__ sval, int *cja,
                              double *cval) {
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < nc;
         c += gridDim.x * blockDim.x) {
        const int src = off[c], dst = cia[c], m = cia[c + 1] - cia[c];
        for (int t = 0; t < m; ++t) {
            cja[dst + t] = scol[src + t];
            cval[dst + t] = sval[src + t];
        }
    }
}

// The same slot lists by a warp per coarse row, without scratch: one pass
// counts a row's slots, and after the scan of the counts a second one forms
// the row and writes it in place (5.4 GB at the 256^3 fine level against 7.2
// for one pass through scratch and a compaction).  The row's entries are taken
// 32 at a time, whatever fine rows they come from.  Lanes with the same coarse
// column find each other with a match; the first of them finds the column's
// slot (a small hash table in shared memory, which a row of at most 32 entries
// does not need), columns seen for the first time take slots in lane order,
// and the first lane adds the values of its group in lane order to the slot.
// Slot numbers and every sum are those of the loop above, bit for bit.  Taking
// the entries one by one (two ballots each) had cost 12.3 ms at that level,
// the compaction by a thread per row 2.4.
// A row whose bound (1 + its entries) exceeds CAP goes to a list for the next
// instantiation; list 2 (above RAP_CAP2) is left to k_rap_build_big.
constexpr int RAP_CAP0 = 64, RAP_CAP1 = 256, RAP_CAP2 = 2048;

template <int CAP>
struct RapTable {
    int key[2 * CAP];               // coarse column, -1 free
    unsigned short slot[2 * CAP];
    int col[CAP];
    double val[CAP];
};

// Sum, in lane order, of the values of the group that this lane leads (mask:
// its lanes; 0 for the others), added to acc.
__device__ __forceinline__ double rap_group_sum(unsigned mask, double acc, double v) {
    const int most = __reduce_max_sync(0xffffffffu, __popc(mask));
    for (int r = 0; r < most; ++r) {
        const double x = __shfl_sync(0xffffffffu, v, __ffs(mask) - 1);
        if (mask) acc += x;
        mask &= mask - 1u;
    }
    return acc;
}

// entry t of a batch of nf <= 32 fine rows (lane q: row q from entry b on,
// `start` entries before it)
__device__ __forceinline__ int rap_entry(int t, int nf, int b, int start) {
    int base = 0;
    for (int r = 0; r < nf; ++r) {
        const int sr = __shfl_sync(0xffffffffu, start, r), br = __shfl_sync(0xffffffffu, b, r);
        if (t >= sr) base = br - sr;
    }
    return base + t;
}

// inclusive sums of len over the lanes
__device__ __forceinline__ int rap_lane_sums(int len) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, len, o);
        if (lane >= o) len += y;
    }
    return len;
}

// Coarse row c of at most 32 entries (m) from nf <= 32 fine rows: the slot
// count, after writing the row (FILL).
template <bool FILL>
__device__ __forceinline__ int rap_short_row(int c, int m, int nf, int b, int start,
                                             const int *__restrict__ ja,
                                             const double *__restrict__ a,
                                             const int *__restrict__ agg, int *cols,
                                             double *vals) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int k = rap_entry(lane, nf, b, start);
    int cc = -1;
    double v = 0.0;
    if (lane < m) {
        cc = agg[ja[k]];
        if (FILL) v = a[k];
    }
    const unsigned grp = __match_any_sync(FULL, cc);
    const bool lead = cc >= 0 && lane == __ffs(grp) - 1;
    const unsigned fresh = __ballot_sync(FULL, lead && cc != c);
    if (FILL) {
        const bool self = lead && cc == c;
        const double acc = rap_group_sum(lead ? grp & (grp - 1u) : 0u, self ? 0.0 + v : v, v);
        const int slot = self ? 0 : 1 + __popc(fresh & ((1u << lane) - 1u));
        if (lead) {
            cols[slot] = cc;
            vals[slot] = acc;
        }
        // the diagonal slot is there even when no entry maps to it
        if (!__any_sync(FULL, self) && lane == 0) {
            cols[0] = c;
            vals[0] = 0.0;
        }
    }
    return 1 + __popc(fresh);
}

// Any other coarse row c, from the fine rows rja[q0, q1) (the first batch's
// b and len at hand), through the table.
template <int CAP, bool FILL>
__device__ __forceinline__ int rap_row(int c, int q0, int q1, int b, int len, RapTable<CAP> *T,
                                       const int *__restrict__ rja, const int *__restrict__ ia,
                                       const int *__restrict__ ja, const double *__restrict__ a,
                                       const int *__restrict__ agg, int *cols, double *vals) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    constexpr unsigned HM = 2 * CAP - 1;
    auto hash = [](int col) { return ((unsigned)col * 2654435761u >> 7) & HM; };
    int cnt = 1;
    for (int t = lane; t < 2 * CAP; t += 32) T->key[t] = -1;
    __syncwarp();
    if (lane == 0) {
        T->key[hash(c)] = c;
        T->slot[hash(c)] = 0;
        T->col[0] = c;
        T->val[0] = 0.0;
    }
    __syncwarp();
    for (int qb = q0; qb < q1; qb += 32) {
        const int nf = min(32, q1 - qb);
        if (qb > q0) {
            b = len = 0;
            if (lane < nf) {
                const int i = rja[qb + lane];
                b = ia[i];
                len = ia[i + 1] - b;
            }
        }
        const int end = rap_lane_sums(len);
        const int m = __shfl_sync(FULL, end, 31);
        for (int tb = 0; tb < m; tb += 32) {
            const int k = rap_entry(tb + lane, nf, b, end - len);
            int cc = -1;
            double v = 0.0;
            if (tb + lane < m) {
                cc = agg[ja[k]];
                if (FILL) v = a[k];
            }
            const unsigned grp = __match_any_sync(FULL, cc);
            const bool lead = cc >= 0 && lane == __ffs(grp) - 1;
            int slot = -1;
            unsigned h = 0;
            if (lead) {
                h = hash(cc);
                for (int key; (key = T->key[h]) != -1; h = (h + 1) & HM)
                    if (key == cc) { slot = T->slot[h]; break; }
            }
            const bool fresh = lead && slot < 0;
            const unsigned nb = __ballot_sync(FULL, fresh);
            if (fresh) {            // distinct columns: only a place can be contended
                slot = cnt + __popc(nb & ((1u << lane) - 1u));
                while (atomicCAS(&T->key[h], -1, cc) != -1) h = (h + 1) & HM;
                T->slot[h] = (unsigned short)slot;
            }
            cnt += __popc(nb);
            if (FILL) {
                const double acc = rap_group_sum(lead ? grp & (grp - 1u) : 0u,
                                                 lead && !fresh ? T->val[slot] + v : v, v);
                if (lead) {
                    T->col[slot] = cc;
                    T->val[slot] = acc;
                }
            }
            __syncwarp();
        }
    }
    if (FILL) {
        for (int t = lane; t < cnt; t += 32) {
            cols[t] = T->col[t];
            vals[t] = T->val[t];
        }
        __syncwarp();
    }
    return cnt;
}

// All rows (CAP = RAP_CAP0), or the rows of list `tier` - 1 (nrow of them,
// read on the device).  list: the rows for the next instantiations, nc each;
// ctl[t]: their number.
template <int CAP, int WARPS, bool FILL, bool LISTED>
__global__ void __launch_bounds__(32 * WARPS, 32 / WARPS)
k_rap_rows(int nc, const int *__restrict__ ria, const int *__restrict__ rja,
           const int *__restrict__ ia, const int *__restrict__ ja, const double *__restrict__ a,
           const int *__restrict__ agg, const int *__restrict__ cia, int *rowcnt, int *cja,
           double *cval, int *list, int *ctl, int tier) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    RapTable<CAP> *T = reinterpret_cast<RapTable<CAP> *>(smem_raw) + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    const int warps = gridDim.x * WARPS;
    const int *mine = list + (size_t)(tier - 1) * nc;
    const int nrow = LISTED ? ctl[tier - 1] : nc;
    // A row's metadata is a chain of three loads (ria, rja, ia), each issued one
    // row ahead of the load that needs it, so that none of them is waited for.
    int c1 = 0, c2 = 0, c3 = 0, p1 = 0, p2 = 0, p3 = 0, n1 = 0, n2 = 0, n3 = 0;
    int i2 = 0, b1 = 0, e1 = 0;
    auto advance = [&](int at) {    // at: the row whose pointers are loaded now
        c1 = c2; p1 = p2; n1 = n2;
        b1 = e1 = 0;
        if (p1 + lane < n1) { b1 = ia[i2]; e1 = ia[i2 + 1]; }
        c2 = c3; p2 = p3; n2 = n3;
        i2 = p2 + lane < n2 ? rja[p2 + lane] : 0;
        p3 = n3 = 0;
        if (at < nrow) {
            c3 = LISTED ? mine[at] : at;
            p3 = ria[c3];
            n3 = ria[c3 + 1];
        }
    };
    int at = blockIdx.x * WARPS + (threadIdx.x >> 5);
    advance(at);
    advance(at + warps);
    advance(at + 2 * warps);
    for (; at < nrow; at += warps) {
        const int cc = c1, r0 = p1, r1 = n1, rb = b1, rl = e1 - b1;
        advance(at + 3 * warps);
        const int end = rap_lane_sums(rl);
        const int m = __shfl_sync(0xffffffffu, end, 31);
        int ub = 1 + m;
        for (int qb = r0 + 32; qb < r1; qb += 32) {
            int l = 0;
            if (qb + lane < r1) {
                const int i = rja[qb + lane];
                l = ia[i + 1] - ia[i];
            }
            ub += __reduce_add_sync(0xffffffffu, l);
        }
        if (ub > CAP) {
            // counted and listed by the count pass; the fill pass leaves it too
            if (!FILL && lane == 0) {
                const int k = ub <= RAP_CAP1 ? 0 : ub <= RAP_CAP2 ? 1 : 2;
                if (!LISTED) list[(size_t)k * nc + atomicAdd(ctl + k, 1)] = cc;
                if (k == 2) rowcnt[cc] = 0;
            }
            continue;
        }
        int *cols = FILL ? cja + cia[cc] : nullptr;
        double *vals = FILL ? cval + cia[cc] : nullptr;
        int cnt;
        if (!LISTED && m <= 32 && r1 - r0 <= 32)
            cnt = rap_short_row<FILL>(cc, m, r1 - r0, rb, end - rl, ja, a, agg, cols, vals);
        else
            cnt = rap_row<CAP, FILL>(cc, r0, r1, rb, rl, T, rja, ia, ja, a, agg, cols, vals);
        if (!FILL && lane == 0) rowcnt[cc] = cnt;
    }
}

// Rows with a bound above RAP_CAP2, a warp each, slots in scratch at off[c]: the
// entries one by one in order, each column looked for by all lanes.  (A thread a
// row, a list of nothing but long rows took 1074 ms where 941 had been spread
// over all rows' warps: HEC aggregates of a random graph of 60 entries a row;
// 43 now.)
__global__ void __launch_bounds__(128)
k_rap_build_big(const int *__restrict__ ria, const int *__restrict__ rja,
                const int *__restrict__ ia, const int *__restrict__ ja,
                const double *__restrict__ a, const int *__restrict__ agg,
                const int *__restrict__ off, const int *__restrict__ list, int nlist, int *scol,
                double *sval, int *rowcnt) {
    constexpr int B = 4;            // places that a lane looks at together
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nlist; t += warps) {
        const int c = list[t];
        int *cols = scol + off[c];
        double *vals = sval + off[c];
        int cnt = 1;
        if (lane == 0) {
            cols[0] = c;
            vals[0] = 0.0;
        }
        __syncwarp();
        for (int q = ria[c]; q < ria[c + 1]; ++q) {
            const int k1 = ia[rja[q] + 1];
            for (int kb = ia[rja[q]]; kb < k1; kb += 32) {
                const int mine = kb + lane < k1 ? agg[ja[kb + lane]] : -1;
                const double v = kb + lane < k1 ? a[kb + lane] : 0.0;
                for (int j = 0; j < min(32, k1 - kb); ++j) {
                    const int cc = __shfl_sync(FULL, mine, j);
                    const double x = __shfl_sync(FULL, v, j);
                    if (cc < 0) continue;
                    int pos = -1;
                    for (int u0 = 0; u0 < cnt && pos < 0; u0 += 32 * B) {
                        int at[B];
#pragma unroll
                        for (int w = 0; w < B; ++w) {
                            const int u = u0 + 32 * w + lane;
                            at[w] = u < cnt ? cols[u] : -1;
                        }
#pragma unroll
                        for (int w = 0; w < B; ++w) {
                            const unsigned hit = __ballot_sync(FULL, at[w] == cc);
                            if (hit) pos = u0 + 32 * w + __ffs(hit) - 1;
                        }
                    }
                    if (lane == 0) {
                        if (pos >= 0) {
                            vals[pos] += x;
                        } else {
                            cols[cnt] = cc;
                            vals[cnt] = x;
                        }
                    }
                    if (pos < 0) ++cnt;
                    __syncwarp();
                }
            }
        }
        if (lane == 0) rowcnt[c] = cnt;
    }
}
// and their rows copied to the product, a warp each
__global__ void k_rap_copy_big(const int *__restrict__ list, int nlist,
                               const int *__restrict__ off, const int *__restrict__ cia,
                               const int *__restrict__ scol, const double *__restrict__ sval,
                               int *cja, double *cval) {
    for (int t = blockIdx.x; t < nlist; t += gridDim.x) {
        const int c = list[t], src = off[c], dst = cia[c], m = cia[c + 1] - dst;
        for (int u = threadIdx.x; u < m; u += blockDim.x) {
            cja[dst + u] = scol[src + u];
            cval[dst + u] = sval[src + u];
        }
    }
}

int rap_agg(const DCsr<double> &A, int nc, const int *agg, const int *ria,
            const int *rja, int **cia_out, int **cja_out, double **cval_out,
            int *cnnz, cudaStream_t s) {
    *cia_out = nullptr; *cja_out = nullptr; *cval_out = nullptr;
    int *tmp = nullptr, *rowcnt = nullptr, *list = nullptr, *ctl = nullptr;
    int *ub = nullptr, *off = nullptr, *scol = nullptr, *cia = nullptr, *cja = nullptr;
    double *sval = nullptr, *cval = nullptr;
    int rc = SUCCESS, h[4] = {0, 0, 0, 0};
    cudaError_t e;
    constexpr int W0 = 8, W1 = 4, W2 = 1;   // warps per CTA of the instantiations
    constexpr size_t S0 = W0 * sizeof(RapTable<RAP_CAP0>), S1 = W1 * sizeof(RapTable<RAP_CAP1>),
                     S2 = W2 * sizeof(RapTable<RAP_CAP2>);
    static bool attr = false;
    if (!attr) {
        cudaFuncSetAttribute(k_rap_rows<RAP_CAP2, W2, false, true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S2);
        cudaFuncSetAttribute(k_rap_rows<RAP_CAP2, W2, true, true>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S2);
        attr = true;
    }
    const int g0 = grid_for(32LL * nc), g1 = std::min(div_up(nc, W1), 4 * sm_count()),
              g2 = std::min(nc, 4 * sm_count());
    if ((rc = dalloc(&tmp, scan_tmp_size(nc + 1)))) goto fail;
    if ((rc = dalloc(&rowcnt, nc))) goto fail;
    if ((rc = dalloc(&list, (size_t)3 * nc))) goto fail;
    if ((rc = dalloc(&ctl, 4))) goto fail;
    if ((rc = dalloc(&cia, nc + 1))) goto fail;
    e = cudaMemsetAsync(ctl, 0, 4 * sizeof(int), s);
    if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto fail; }
    k_rap_rows<RAP_CAP0, W0, false, false><<<g0, 32 * W0, S0, s>>>(
        nc, ria, rja, A.ia, A.ja, A.val, agg, nullptr, rowcnt, nullptr, nullptr, list, ctl, 0);
    k_rap_rows<RAP_CAP1, W1, false, true><<<g1, 32 * W1, S1, s>>>(
        nc, ria, rja, A.ia, A.ja, A.val, agg, nullptr, rowcnt, nullptr, nullptr, list, ctl, 1);
    k_rap_rows<RAP_CAP2, W2, false, true><<<g2, 32 * W2, S2, s>>>(
        nc, ria, rja, A.ia, A.ja, A.val, agg, nullptr, rowcnt, nullptr, nullptr, list, ctl, 2);
    count_launch(3);
    if ((rc = scan_exclusive(rowcnt, cia, nc, tmp, s))) goto fail;
    e = cudaMemcpyAsync(ctl + 3, cia + nc, sizeof(int), cudaMemcpyDeviceToDevice, s);
    if (e == cudaSuccess) e = cudaMemcpyAsync(h, ctl, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto fail; }
    if (h[2]) {
        // rows of thousands of entries: bounds, scratch and a warp per row
        int total = 0;
        if ((rc = dalloc(&ub, nc))) goto fail;
        if ((rc = dalloc(&off, nc + 1))) goto fail;
        k_rap_bound<<<grid_for(nc), 256, 0, s>>>(nc, ria, rja, A.ia, ub);
        count_launch();
        if ((rc = scan_exclusive(ub, off, nc, tmp, s))) goto fail;
        e = cudaMemcpyAsync(&total, off + nc, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto fail; }
        if ((rc = dalloc(&scol, total))) goto fail;
        if ((rc = dalloc(&sval, total))) goto fail;
        k_rap_build_big<<<grid_for(32LL * h[2], 128), 128, 0, s>>>(
            ria, rja, A.ia, A.ja, A.val, agg, off, list + (size_t)2 * nc, h[2], scol, sval, rowcnt);
        count_launch();
        if ((rc = scan_exclusive(rowcnt, cia, nc, tmp, s))) goto fail;
        e = cudaMemcpyAsync(&h[3], cia + nc, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto fail; }
    }
    *cnnz = h[3];
    if ((rc = dalloc(&cja, *cnnz))) goto fail;
    if ((rc = dalloc(&cval, *cnnz))) goto fail;
    k_rap_rows<RAP_CAP0, W0, true, false><<<g0, 32 * W0, S0, s>>>(
        nc, ria, rja, A.ia, A.ja, A.val, agg, cia, rowcnt, cja, cval, list, ctl, 0);
    count_launch();
    if (h[0]) {
        k_rap_rows<RAP_CAP1, W1, true, true><<<std::min(div_up(h[0], W1), g1), 32 * W1, S1, s>>>(
            nc, ria, rja, A.ia, A.ja, A.val, agg, cia, rowcnt, cja, cval, list, ctl, 1);
        count_launch();
    }
    if (h[1]) {
        k_rap_rows<RAP_CAP2, W2, true, true><<<std::min(h[1], g2), 32 * W2, S2, s>>>(
            nc, ria, rja, A.ia, A.ja, A.val, agg, cia, rowcnt, cja, cval, list, ctl, 2);
        count_launch();
    }
    if (h[2]) {
        k_rap_copy_big<<<std::min(h[2], 4 * sm_count()), 128, 0, s>>>(
            list + (size_t)2 * nc, h[2], off, cia, scol, sval, cja, cval);
        count_launch();
    }
    e = cudaGetLastError();
    if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto fail; }
    dfree(tmp); dfree(rowcnt); dfree(list); dfree(ctl);
    dfree(ub); dfree(off); dfree(scol); dfree(sval);
    *cia_out = cia; *cja_out = cja; *cval_out = cval;
    return SUCCESS;
fail:
    dfree(tmp); dfree(rowcnt); dfree(list); dfree(ctl);
    dfree(ub); dfree(off); dfree(scol); dfree(sval);
    dfree(cia); dfree(cja); dfree(cval);
    return rc;
}

// ---------------------------------------------------------------------------
// smoother diagonals
// ---------------------------------------------------------------------------
__global__ void k_diags(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                        const double *__restrict__ a, double *djac, double *dgs,
                        double *dsor, int *gs_ok, int *sor_ok, int *missing) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        double dj = 0.0, dg = 0.0, ds = 0.0;
        int okg = 0, oks = 0;
        for (int k = ia[i]; k < ia[i + 1]; ++k) {
            if (ja[k] != i) continue;
            dj = a[k];
            ds = a[k];
            oks = 1;
            if (fabs(a[k]) > SMALLREAL) { dg = 1.e+0 / a[k]; okg = 1; }
        }
        djac[i] = dj;
        dgs[i] = dg;
        dsor[i] = ds;
        gs_ok[i] = okg;
        sor_ok[i] = oks;
        if (!okg || !oks) atomicAdd(missing, 1);
    }
}

// Rows without a (usable) diagonal keep the previous row's d in the
// reference's sweep; resolve that carry sequentially (rare path).
__global__ void k_diag_carry(int n, const double *__restrict__ dgs,
                             const double *__restrict__ dsor,
                             const int *__restrict__ gs_ok,
                             const int *__restrict__ sor_ok, double *gf,
                             double *gb, double *sf, double *sb) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double c1 = 0.0, c2 = 0.0;
    for (int i = 0; i < n; ++i) {
        if (gs_ok[i]) c1 = dgs[i];
        if (sor_ok[i]) c2 = dsor[i];
        gf[i] = c1;
        sf[i] = c2;
    }
    c1 = 0.0; c2 = 0.0;
    for (int i = n - 1; i >= 0; --i) {
        if (gs_ok[i]) c1 = dgs[i];
        if (sor_ok[i]) c2 = dsor[i];
        gb[i] = c1;
        sb[i] = c2;
    }
}

int smoother_diagonals(const DCsr<double> &A, double *d_jac, double *d_gs_f,
                       double *d_gs_b, double *d_sor_f, double *d_sor_b,
                       cudaStream_t s) {
    const int n = A.n;
    int *ok = nullptr;
    HZB_TRY(dalloc(&ok, 2 * (size_t)n + 1));
    int *missing = ok + 2 * (size_t)n;
    HZB_CUDA(cudaMemsetAsync(missing, 0, sizeof(int), s));
    k_diags<<<grid_for(n), 256, 0, s>>>(n, A.ia, A.ja, A.val, d_jac, d_gs_f, d_sor_f,
                                        ok, ok + n, missing);
    count_launch();
    int h = 0;
    cudaError_t e = cudaMemcpyAsync(&h, missing, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { dfree(ok); set_error(e, __FILE__, __LINE__); return ERROR_SOLVER_MISC; }
    if (h) {
        double *tg = nullptr, *ts = nullptr;
        int rc = dalloc(&tg, n);
        if (!rc) rc = dalloc(&ts, n);
        if (rc) { dfree(tg); dfree(ok); return rc; }
        cudaMemcpyAsync(tg, d_gs_f, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(ts, d_sor_f, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
        k_diag_carry<<<1, 32, 0, s>>>(n, tg, ts, ok, ok + n, d_gs_f, d_gs_b, d_sor_f,
                                      d_sor_b);
        count_launch();
        e = cudaStreamSynchronize(s);
        dfree(tg); dfree(ts);
        if (e != cudaSuccess) { dfree(ok); set_error(e, __FILE__, __LINE__); return ERROR_SOLVER_MISC; }
    } else {
        cudaMemcpyAsync(d_gs_b, d_gs_f, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
        cudaMemcpyAsync(d_sor_b, d_sor_f, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
    }
    dfree(ok);
    HZB_LAUNCH_CHECK();
    return SUCCESS;
}

// ---------------------------------------------------------------------------
// A^T with ascending column indices per row (dcsr_transz, p = NULL)
// ---------------------------------------------------------------------------
__global__ void k_tr_count(int n, const int *__restrict__ ia,
                           const int *__restrict__ ja, int *cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        for (int k = ia[i]; k < ia[i + 1]; ++k) atomicAdd(cnt + ja[k], 1);
}
__global__ void k_tr_fill(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                          const double *__restrict__ a, const int *__restrict__ tia,
                          int *fillc, int *tja, double *tval) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        for (int k = ia[i]; k < ia[i + 1]; ++k) {
            const int q = tia[ja[k]] + atomicAdd(fillc + ja[k], 1);
            tja[q] = i;
            tval[q] = a[k];
        }
}
// rows of the transpose in ascending order (stable for equal indices is not
// needed: a row index appears once per source row entry)
__global__ void k_tr_sort(int n, const int *__restrict__ tia, int *tja, double *tval) {
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < n;
         r += gridDim.x * blockDim.x) {
        const int b0 = tia[r], b1 = tia[r + 1];
        for (int p = b0 + 1; p < b1; ++p) {
            const int v = tja[p];
            const double x = tval[p];
            int q = p - 1;
            while (q >= b0 && tja[q] > v) { tja[q + 1] = tja[q]; tval[q + 1] = tval[q]; --q; }
            tja[q + 1] = v;
            tval[q + 1] = x;
        }
    }
}

int transpose_csr(const DCsr<double> &A, int **tia_out, int **tja_out,
                  double **tval_out, cudaStream_t s) {
    const int n = A.n;
    int *tia = nullptr, *tja = nullptr, *cnt = nullptr, *tmp = nullptr;
    double *tval = nullptr;
    int rc = SUCCESS;
    const int g = grid_for(n);
    if ((rc = dalloc(&tia, n + 1)) || (rc = dalloc(&tja, A.nnz)) ||
        (rc = dalloc(&tval, A.nnz)) || (rc = dalloc(&cnt, n)) ||
        (rc = dalloc(&tmp, scan_tmp_size(n + 1)))) goto fail;
    cudaMemsetAsync(cnt, 0, sizeof(int) * n, s);
    k_tr_count<<<g, 256, 0, s>>>(n, A.ia, A.ja, cnt);
    count_launch();
    if ((rc = scan_exclusive(cnt, tia, n, tmp, s))) goto fail;
    cudaMemsetAsync(cnt, 0, sizeof(int) * n, s);
    k_tr_fill<<<g, 256, 0, s>>>(n, A.ia, A.ja, A.val, tia, cnt, tja, tval);
    k_tr_sort<<<g, 256, 0, s>>>(n, tia, tja, tval);
    count_launch(2);
    if (cudaStreamSynchronize(s) != cudaSuccess) {
        set_error(cudaGetLastError(), __FILE__, __LINE__);
        rc = ERROR_SOLVER_MISC;
        goto fail;
    }
    dfree(cnt); dfree(tmp);
    *tia_out = tia; *tja_out = tja; *tval_out = tval;
    return SUCCESS;
fail:
    dfree(tia); dfree(tja); dfree(tval); dfree(cnt); dfree(tmp);
    return rc;
}

// ---------------------------------------------------------------------------
// level schedules (Kahn rounds on the DAG lower -> higher or reverse)
// ---------------------------------------------------------------------------
void Schedule::release() {
    dfree(rows);
    dfree(set_ptr);
    dfree(bar);
    stream.release();
    h_ptr.clear();
    run_first.clear();
    run_last.clear();
    run_max.clear();
}

__global__ void k_transpose_count(int n, const int *__restrict__ ia,
                                  const int *__restrict__ ja, int *cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        for (int k = ia[i]; k < ia[i + 1]; ++k) atomicAdd(cnt + ja[k], 1);
}
__global__ void k_transpose_fill(int n, const int *__restrict__ ia,
                                 const int *__restrict__ ja,
                                 const int *__restrict__ tia, int *fillc, int *tja) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        for (int k = ia[i]; k < ia[i + 1]; ++k) {
            const int j = ja[k];
            tja[tia[j] + atomicAdd(fillc + j, 1)] = i;
        }
}

// dependency count: neighbours that come earlier in the sweep
__global__ void k_indeg(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                        const int *__restrict__ tia, const int *__restrict__ tja,
                        int *indeg, int *rows, int *tail) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        int c = 0;
        for (int k = ia[i]; k < ia[i + 1]; ++k) {
            const int j = ja[k];
            c += j < i;
        }
        for (int k = tia[i]; k < tia[i + 1]; ++k) {
            const int j = tja[k];
            c += j < i;
        }
        indeg[i] = c;
        atomicMax(tail + 1, c);
        if (c == 0) rows[atomicAdd(tail, 1)] = i;
    }
}

__global__ void k_kahn_round(int head, int cnt, const int *__restrict__ ia,
                             const int *__restrict__ ja, const int *__restrict__ tia,
                             const int *__restrict__ tja, int *indeg,
                             int *rows, int *tail) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < cnt;
         q += gridDim.x * blockDim.x) {
        const int i = rows[head + q];
        for (int k = ia[i]; k < ia[i + 1]; ++k) {
            const int j = ja[k];
            if (j > i)
                if (atomicSub(indeg + j, 1) == 1) rows[atomicAdd(tail, 1)] = j;
        }
        for (int k = tia[i]; k < tia[i + 1]; ++k) {
            const int j = tja[k];
            if (j > i)
                if (atomicSub(indeg + j, 1) == 1) rows[atomicAdd(tail, 1)] = j;
        }
    }
}

// Every round of Kahn's algorithm in one CTA: the frontier [head, cur) of the
// queue releases the rows that depend on it; the queue end moves by a
// shared-memory atomic and the rounds are separated by __syncthreads, so a
// level of many small sets costs no launch or host round trip per set.
// Each round removes at least one row, so at most n rounds run.  ptr
// receives the set boundaries (n + 1 ints at most), *nsets their count.
constexpr int KAHN_CTA_MAX_ROWS = 1 << 20;
__global__ void __launch_bounds__(1024)
k_kahn_all(int n, const int *__restrict__ ia, const int *__restrict__ ja,
           const int *__restrict__ tia, const int *__restrict__ tja,
           int *indeg, int *rows, const int *__restrict__ tail0, int *ptr, int *nsets) {
    __shared__ int s_tail, s_head, s_cur, s_ns;
    if (threadIdx.x == 0) {
        s_head = 0;
        s_cur = *tail0;
        s_tail = s_cur;
        s_ns = 0;
        ptr[0] = 0;
    }
    __syncthreads();
    for (int round = 0; round < n; ++round) {
        const int head = s_head, cur = s_cur;
        if (cur <= head) break;
        if (threadIdx.x == 0) ptr[++s_ns] = cur;
        for (int q = head + threadIdx.x; q < cur; q += blockDim.x) {
            const int i = rows[q];
            for (int k = ia[i]; k < ia[i + 1]; ++k) {
                const int j = ja[k];
                if (j > i)
                    if (atomicSub(indeg + j, 1) == 1) rows[atomicAdd(&s_tail, 1)] = j;
            }
            for (int k = tia[i]; k < tia[i + 1]; ++k) {
                const int j = tja[k];
                if (j > i)
                    if (atomicSub(indeg + j, 1) == 1) rows[atomicAdd(&s_tail, 1)] = j;
            }
        }
        __threadfence_block();
        __syncthreads();
        if (threadIdx.x == 0) {
            s_head = cur;
            s_cur = s_tail;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        nsets[0] = s_ns;
        nsets[1] = s_head;   // rows placed
    }
}

// The same rounds for levels of at most KAHN_SMEM_ROWS rows whose in-degrees
// fit 16 bits: the in-degree counters sit in shared memory (two to a word;
// a counter is decremented exactly as often as it counts, so a halfword
// never borrows from its neighbour), and each round's new frontier is also
// kept in shared memory (double-buffered, up to KAHN_FRONT rows) for the next
// round to read, so a round costs two dependent global loads (row bounds,
// then columns) instead of a chain through global atomics.  The column
// indices of a row are loaded eight at a time before their counters are
// decremented.  Same sets as k_kahn_all (the order of rows inside a set may
// differ; the rows of a set are independent).
constexpr int KAHN_SMEM_ROWS = 96 * 1024;
constexpr int KAHN_FRONT = 4096;
constexpr size_t kahn_smem_bytes(int n) {
    return sizeof(unsigned) * ((size_t)(n + 1) / 2) + sizeof(int) * 2 * KAHN_FRONT;
}
__global__ void __launch_bounds__(1024)
k_kahn_smem(int n, const int *__restrict__ ia, const int *__restrict__ ja,
            const int *__restrict__ tia, const int *__restrict__ tja,
            const int *__restrict__ indeg, int *rows, const int *__restrict__ tail0, int *ptr,
            int *nsets) {
    extern __shared__ unsigned kahn_sm[];
    const int nw = (n + 1) / 2;
    unsigned *deg = kahn_sm;
    int *front = reinterpret_cast<int *>(kahn_sm + nw);
    __shared__ int s_tail, s_head, s_cur, s_ns;
    for (int w = threadIdx.x; w < nw; w += blockDim.x) {
        const unsigned lo = (unsigned)indeg[2 * w];
        const unsigned hi = 2 * w + 1 < n ? (unsigned)indeg[2 * w + 1] : 0u;
        deg[w] = lo | (hi << 16);
    }
    if (threadIdx.x == 0) {
        s_head = 0;
        s_cur = *tail0;
        s_tail = s_cur;
        s_ns = 0;
        ptr[0] = 0;
    }
    __syncthreads();
    for (int round = 0; round < n; ++round) {
        const int head = s_head, cur = s_cur;
        if (cur <= head) break;
        if (threadIdx.x == 0) ptr[++s_ns] = cur;
        const bool fin_ok = round > 0 && cur - head <= KAHN_FRONT;
        const int *fin = front + (round & 1) * KAHN_FRONT;
        int *fout = front + ((round + 1) & 1) * KAHN_FRONT;
        auto release = [&](int j) {
            const unsigned sh = 16u * (unsigned)(j & 1);
            const unsigned old = atomicSub(deg + (j >> 1), 1u << sh);
            if (((old >> sh) & 0xFFFFu) == 1u) {
                const int p = atomicAdd(&s_tail, 1);
                rows[p] = j;
                if (p - cur < KAHN_FRONT) fout[p - cur] = j;
            }
        };
        auto visit = [&](int i, const int *__restrict__ xa, const int *__restrict__ xj) {
            const int k1 = xa[i + 1];
            for (int k0 = xa[i]; k0 < k1; k0 += 8) {
                int c[8];
#pragma unroll
                for (int u = 0; u < 8; ++u) c[u] = k0 + u < k1 ? xj[k0 + u] : -1;
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    if (c[u] >= 0 && c[u] > i) release(c[u]);
            }
        };
        for (int q = head + threadIdx.x; q < cur; q += blockDim.x) {
            const int i = fin_ok ? fin[q - head] : rows[q];
            visit(i, ia, ja);
            visit(i, tia, tja);
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            s_head = cur;
            s_cur = s_tail;
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        nsets[0] = s_ns;
        nsets[1] = s_head;   // rows placed
    }
}

static void make_runs(Schedule *sch) {
    const int ns = (int)sch->h_ptr.size() - 1;
    int k = 0;
    while (k < ns) {
        int k2 = k;
        int mx = 0;
        while (k2 < ns && k2 - k < GS_RUN_SETS &&
               sch->h_ptr[k2 + 1] - sch->h_ptr[k2] <= GS_SMALL_SET) {
            mx = std::max(mx, sch->h_ptr[k2 + 1] - sch->h_ptr[k2]);
            ++k2;
        }
        if (k2 > k) {   // run of small sets
            sch->run_first.push_back(k);
            sch->run_last.push_back(k2);
            sch->run_max.push_back(mx);
            k = k2;
        } else {        // one large set: a grid-wide launch (marked by -1)
            sch->run_first.push_back(k);
            sch->run_last.push_back(-1);
            sch->run_max.push_back(sch->h_ptr[k + 1] - sch->h_ptr[k]);
            ++k;
        }
    }
}

int gs_schedule(int n, const int *ia, const int *ja, int nnz,
                Schedule *sch, cudaStream_t s) {
    sch->release();
    int *tia = nullptr, *tja = nullptr, *fillc = nullptr, *indeg = nullptr;
    int *tail = nullptr, *tmp = nullptr;
    int rc = SUCCESS;
    std::vector<int> ptr;
    cudaError_t e;
    const int g = grid_for(n);
    if ((rc = dalloc(&tia, n + 1))) goto done;
    if ((rc = dalloc(&tja, nnz))) goto done;
    if ((rc = dalloc(&fillc, n))) goto done;
    if ((rc = dalloc(&indeg, n))) goto done;
    if ((rc = dalloc(&tail, 2))) goto done;   // frontier end, largest in-degree
    if ((rc = dalloc(&tmp, scan_tmp_size(n + 1)))) goto done;
    if ((rc = dalloc(&sch->rows, n))) goto done;
    cudaMemsetAsync(fillc, 0, sizeof(int) * n, s);
    cudaMemsetAsync(tail, 0, 2 * sizeof(int), s);
    k_transpose_count<<<g, 256, 0, s>>>(n, ia, ja, fillc);
    count_launch();
    if ((rc = scan_exclusive(fillc, tia, n, tmp, s))) goto done;
    cudaMemsetAsync(fillc, 0, sizeof(int) * n, s);
    k_transpose_fill<<<g, 256, 0, s>>>(n, ia, ja, tia, fillc, tja);
    k_indeg<<<g, 256, 0, s>>>(n, ia, ja, tia, tja, indeg, sch->rows, tail);
    count_launch(2);
    if (n <= KAHN_CTA_MAX_ROWS) {
        // one CTA runs every round; set boundaries and counts come back once
        int *dptr = nullptr, *dns = nullptr;
        if ((rc = dalloc(&dptr, n + 1)) || (rc = dalloc(&dns, 2))) {
            dfree(dptr);
            goto done;
        }
        int maxdeg = 0;
        e = cudaMemcpyAsync(&maxdeg, tail + 1, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            dfree(dptr);
            dfree(dns);
            set_error(e, __FILE__, __LINE__);
            rc = ERROR_SOLVER_MISC;
            goto done;
        }
        if (n <= KAHN_SMEM_ROWS && maxdeg <= 0xFFFF) {
            static bool attr = false;
            if (!attr) {
                cudaFuncSetAttribute(k_kahn_smem, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)kahn_smem_bytes(KAHN_SMEM_ROWS));
                attr = true;
            }
            k_kahn_smem<<<1, 1024, kahn_smem_bytes(n), s>>>(n, ia, ja, tia, tja,
                                                            indeg, sch->rows, tail, dptr, dns);
        } else {
            k_kahn_all<<<1, 1024, 0, s>>>(n, ia, ja, tia, tja, indeg, sch->rows,
                                          tail, dptr, dns);
        }
        count_launch();
        int hns[2] = {0, 0};
        e = cudaMemcpyAsync(hns, dns, sizeof(hns), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e == cudaSuccess && hns[1] == n) {
            ptr.resize(hns[0] + 1);
            e = cudaMemcpyAsync(ptr.data(), dptr, sizeof(int) * (hns[0] + 1),
                                cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        }
        dfree(dptr);
        dfree(dns);
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto done; }
        if (hns[1] != n) {
            set_error_msg("gs_schedule: incomplete level schedule");
            rc = ERROR_DATA_STRUCTURE;
            goto done;
        }
    } else {
        int head = 0, cur = 0;
        e = cudaMemcpyAsync(&cur, tail, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto done; }
        ptr.push_back(0);
        while (cur > head) {
            ptr.push_back(cur);
            const int cnt = cur - head;
            k_kahn_round<<<grid_for(cnt), 256, 0, s>>>(head, cnt, ia, ja, tia, tja,
                                                       indeg, sch->rows, tail);
            count_launch();
            head = cur;
            e = cudaMemcpyAsync(&cur, tail, sizeof(int), cudaMemcpyDeviceToHost, s);
            if (e == cudaSuccess) e = cudaStreamSynchronize(s);
            if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto done; }
        }
        if (head != n) {   // a cycle cannot occur in index order; guard anyway
            set_error_msg("gs_schedule: incomplete level schedule");
            rc = ERROR_DATA_STRUCTURE;
            goto done;
        }
    }
    sch->h_ptr = ptr;
    if ((rc = dalloc(&sch->bar, 2))) goto done;
    if (cudaMemsetAsync(sch->bar, 0, 2 * sizeof(unsigned), s) != cudaSuccess) {
        rc = ERROR_SOLVER_MISC;
        goto done;
    }
    if ((rc = dalloc(&sch->set_ptr, ptr.size()))) goto done;
    e = cudaMemcpyAsync(sch->set_ptr, ptr.data(), sizeof(int) * ptr.size(),
                        cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto done; }
    make_runs(sch);
done:
    dfree(tia); dfree(tja); dfree(fillc); dfree(indeg); dfree(tail); dfree(tmp);
    if (rc) sch->release();
    return rc;
}

__global__ void k_reverse(int n, const int *__restrict__ in, int *out) {
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < n; q += gridDim.x * blockDim.x)
        out[q] = in[n - 1 - q];
}

int gs_schedule_reverse(const Schedule &f, int n, Schedule *sch, cudaStream_t s) {
    sch->release();
    const int ns = (int)f.h_ptr.size() - 1;
    std::vector<int> ptr(ns + 1);
    for (int k = 0; k <= ns; ++k) ptr[k] = n - f.h_ptr[ns - k];
    int rc = SUCCESS;
    if (!(rc = dalloc(&sch->rows, n)) && !(rc = dalloc(&sch->bar, 2)) &&
        !(rc = dalloc(&sch->set_ptr, ptr.size()))) {
        k_reverse<<<grid_for(n), 256, 0, s>>>(n, f.rows, sch->rows);
        count_launch();
        cudaError_t e = cudaMemsetAsync(sch->bar, 0, 2 * sizeof(unsigned), s);
        if (e == cudaSuccess)
            e = cudaMemcpyAsync(sch->set_ptr, ptr.data(), sizeof(int) * ptr.size(),
                                cudaMemcpyHostToDevice, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; }
    }
    if (rc) {
        sch->release();
        return rc;
    }
    sch->h_ptr = ptr;
    make_runs(sch);
    return SUCCESS;
}

// ---------------------------------------------------------------------------
// multicolouring (Jones-Plassmann, hashed priorities, smallest free colour)
// ---------------------------------------------------------------------------

__global__ void k_jp_round(int n, const int *__restrict__ ia, const int *__restrict__ ja,
                           const int *__restrict__ col_in, int *col_out, int *left) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x) {
        int c = col_in[i];
        if (c >= 0) { col_out[i] = c; continue; }
        const unsigned pi = hash_u32((unsigned)i);
        bool top = true;
        unsigned long long used = 0ull;   // colours 0..63 taken by neighbours
        for (int k = ia[i]; k < ia[i + 1]; ++k) {
            const int j = ja[k];
            if (j == i) continue;
            const int cj = col_in[j];
            if (cj >= 0) {
                if (cj < 64) used |= 1ull << cj;
            } else {
                const unsigned pj = hash_u32((unsigned)j);
                if (pj > pi || (pj == pi && j > i)) { top = false; }
            }
        }
        if (top) {
            int cc = 0;
            while (cc < 64 && (used >> cc & 1ull)) ++cc;
            col_out[i] = cc;
        } else {
            col_out[i] = -1;
            atomicAdd(left, 1);
        }
    }
}

__global__ void k_color_count(int n, const int *__restrict__ col, int *cnt) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        atomicAdd(cnt + col[i], 1);
}
__global__ void k_color_fill(int n, const int *__restrict__ col,
                             const int *__restrict__ ptr, int *fillc, int *rows) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += gridDim.x * blockDim.x)
        rows[ptr[col[i]] + atomicAdd(fillc + col[i], 1)] = i;
}

int multicolor(int n, const int *ia, const int *ja, Schedule *sch, cudaStream_t s) {
    sch->release();
    int *c0 = nullptr, *c1 = nullptr, *left = nullptr, *cnt = nullptr, *ptr = nullptr;
    int *tmp = nullptr;
    int rc = SUCCESS, ncol = 0;
    cudaError_t e;
    const int g = grid_for(n);
    std::vector<int> hp;
    if ((rc = dalloc(&c0, n))) goto done;
    if ((rc = dalloc(&c1, n))) goto done;
    if ((rc = dalloc(&left, 1))) goto done;
    if ((rc = dalloc(&cnt, 65))) goto done;
    if ((rc = dalloc(&ptr, 66))) goto done;
    if ((rc = dalloc(&tmp, scan_tmp_size(66)))) goto done;
    if ((rc = dalloc(&sch->rows, n))) goto done;
    cudaMemsetAsync(c0, 0xff, sizeof(int) * n, s);
    for (int round = 0; round < 4096; ++round) {
        int hl = 0;
        cudaMemsetAsync(left, 0, sizeof(int), s);
        k_jp_round<<<g, 256, 0, s>>>(n, ia, ja, c0, c1, left);
        count_launch();
        std::swap(c0, c1);
        e = cudaMemcpyAsync(&hl, left, sizeof(int), cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto done; }
        if (!hl) break;
    }
    cudaMemsetAsync(cnt, 0, sizeof(int) * 65, s);
    k_color_count<<<g, 256, 0, s>>>(n, c0, cnt);
    count_launch();
    if ((rc = scan_exclusive(cnt, ptr, 65, tmp, s))) goto done;
    hp.resize(66);
    e = cudaMemcpyAsync(hp.data(), ptr, sizeof(int) * 66, cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto done; }
    if (hp[65] != n) { set_error_msg("multicolor: more than 64 colours"); rc = ERROR_DATA_STRUCTURE; goto done; }
    cudaMemsetAsync(cnt, 0, sizeof(int) * 65, s);
    k_color_fill<<<g, 256, 0, s>>>(n, c0, ptr, cnt, sch->rows);
    count_launch();
    ncol = 0;
    while (ncol < 65 && hp[ncol + 1] > hp[ncol]) ++ncol;
    sch->h_ptr.assign(hp.begin(), hp.begin() + ncol + 1);
    if ((rc = dalloc(&sch->set_ptr, ncol + 1))) goto done;
    e = cudaMemcpyAsync(sch->set_ptr, sch->h_ptr.data(), sizeof(int) * (ncol + 1),
                        cudaMemcpyHostToDevice, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); rc = ERROR_SOLVER_MISC; goto done; }
    make_runs(sch);
done:
    dfree(c0); dfree(c1); dfree(left); dfree(cnt); dfree(ptr); dfree(tmp);
    if (rc) sch->release();
    return rc;
}

// ---------------------------------------------------------------------------
// Galerkin product without device allocation.
//
// Some callers cannot call cudaMalloc: processes whose device memory is
// reserved up front by their own allocator (a framework's caching pool, an
// embedded solver with a fixed memory budget), and library code that must
// not trigger the implicit device synchronisation that cudaMalloc and
// cudaFree bring.  For them the product's scratch (restriction pattern,
// per-row bounds, slot lists, scan partials, an error flag) lives in one
// file-scope device array of fixed size, held by every device that loads
// this library until the process exits.  Its size bounds the problem:
// n <= HZB_NOALLOC_MAX_ROWS fine rows and nnz <= HZB_NOALLOC_MAX_NNZ stored
// entries.
// ---------------------------------------------------------------------------
namespace {
constexpr size_t NA_ROWS = HZB_NOALLOC_MAX_ROWS;
constexpr size_t NA_NNZ = HZB_NOALLOC_MAX_NNZ;
constexpr size_t NA_TMP = (NA_ROWS + 1 + 2047) / 2048 + 8;
constexpr size_t NA_SLOTS = NA_NNZ + NA_ROWS;   // slot lists: nc + sum of row lengths
// int words: cnt, ria, rja, ub, off, rowcnt, scan tmp, error flag (padded), scol
constexpr size_t NA_INTS = 6 * (NA_ROWS + 1) + NA_TMP + 4 + NA_SLOTS;
constexpr size_t NA_INT_WORDS = (NA_INTS + 1) / 2;   // in 8-byte words
constexpr size_t NA_WORDS = NA_INT_WORDS + NA_SLOTS;   // + sval
}  // namespace

static __device__ __align__(256) double g_noalloc_scratch[NA_WORDS];

// Device address of g_noalloc_scratch for each device, resolved once with
// that device current (in host code the symbol is only a host stand-in).
static void *g_noalloc_addr[64];
static std::mutex g_noalloc_mu;

static int noalloc_scratch(double **p) {
    int dev = 0;
    HZB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) { set_error_msg("device ordinal out of range"); return ERROR_MISC; }
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_addr[dev]) {
        void *a = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&a, g_noalloc_scratch);
        if (e != cudaSuccess) { set_error(e, __FILE__, __LINE__); return ERROR_SOLVER_MISC; }
        g_noalloc_addr[dev] = a;
    }
    *p = (double *)g_noalloc_addr[dev];
    return SUCCESS;
}

}  // namespace hzb

// The same kernels, in the same order, as hzb_rap_agg_device, so the result
// is identical bit for bit; only the scratch comes from the static array and
// the outputs from the caller.  The inputs are checked on the device before
// any kernel indexes by them, and the slot lists' total against the array
// before they are written.
extern "C" INT hzb_rap_agg_device_noalloc(INT n, INT nnz, const INT *ia, const INT *ja,
                                          const REAL *val, INT nc, const INT *agg,
                                          INT cap_nnz, INT *rap_ia, INT *rap_ja,
                                          REAL *rap_val, INT *rap_nnz) {
    using namespace hzb;
    if (n < 1 || nnz < 0 || nc < 1 || nc > n || (size_t)n > NA_ROWS || (size_t)nnz > NA_NNZ) {
        set_error_msg("hzb_rap_agg_device_noalloc: sizes beyond HZB_NOALLOC_MAX_ROWS / "
                      "HZB_NOALLOC_MAX_NNZ");
        return ERROR_MAT_SIZE;
    }
    if (!ia || !ja || !val || !agg || !rap_ia || !rap_nnz || cap_nnz < 0) {
        set_error_msg("hzb_rap_agg_device_noalloc: null array or negative capacity");
        return ERROR_INPUT_PAR;
    }
    double *base = nullptr;
    HZB_TRY(noalloc_scratch(&base));
    int *ip = (int *)base;
    int *cnt = ip;                       ip += NA_ROWS + 1;
    int *ria = ip;                       ip += NA_ROWS + 1;
    int *rja = ip;                       ip += NA_ROWS + 1;
    int *ub = ip;                        ip += NA_ROWS + 1;
    int *off = ip;                       ip += NA_ROWS + 1;
    int *rowcnt = ip;                    ip += NA_ROWS + 1;
    int *tmp = ip;                       ip += NA_TMP;
    int *bad = ip;                       ip += 4;
    int *scol = ip;
    double *sval = base + NA_INT_WORDS;
    cudaStream_t s = 0;
    const int gn = grid_for(n), gc = grid_for(nc);
    HZB_TRY(check_rap_inputs(n, nnz, ia, ja, nc, agg, bad, s));
    // R = P^T (counts start at zero: the array keeps the previous call's data)
    HZB_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * nc, s));
    k_agg_count<<<gn, 256, 0, s>>>(n, agg, cnt);
    count_launch();
    HZB_TRY(scan_exclusive(cnt, ria, nc, tmp, s));
    HZB_CUDA(cudaMemsetAsync(cnt, 0, sizeof(int) * nc, s));
    k_agg_fill<<<gn, 256, 0, s>>>(n, agg, ria, cnt, rja);
    k_sort_rows<<<gc, 256, 0, s>>>(nc, ria, rja);
    // slot lists per coarse row, then the compacted product
    k_rap_bound<<<gc, 256, 0, s>>>(nc, ria, rja, ia, ub);
    count_launch(3);
    HZB_TRY(scan_exclusive(ub, off, nc, tmp, s));
    int slots = 0;
    HZB_CUDA(cudaMemcpyAsync(&slots, off + nc, sizeof(int), cudaMemcpyDeviceToHost, s));
    HZB_CUDA(cudaStreamSynchronize(s));
    if (slots < 0 || (size_t)slots > NA_SLOTS) {
        set_error_msg("hzb_rap_agg_device_noalloc: the slot lists exceed the static scratch");
        return ERROR_MAT_SIZE;
    }
    k_rap_build<<<gc, 128, 0, s>>>(nc, ria, rja, ia, ja, val, agg, off, scol, sval, rowcnt);
    count_launch();
    HZB_TRY(scan_exclusive(rowcnt, rap_ia, nc, tmp, s));
    int total = 0;
    HZB_CUDA(cudaMemcpyAsync(&total, rap_ia + nc, sizeof(int), cudaMemcpyDeviceToHost, s));
    HZB_CUDA(cudaStreamSynchronize(s));
    *rap_nnz = total;
    if (total > cap_nnz) {
        set_error_msg("hzb_rap_agg_device_noalloc: output capacity too small (*rap_nnz "
                      "holds the size needed)");
        return ERROR_INPUT_PAR;
    }
    if (total > 0 && (!rap_ja || !rap_val)) {
        set_error_msg("hzb_rap_agg_device_noalloc: null output array");
        return ERROR_INPUT_PAR;
    }
    k_rap_compact<<<gc, 256, 0, s>>>(nc, off, rap_ia, scol, sval, rap_ja, rap_val);
    count_launch();
    HZB_CUDA(cudaStreamSynchronize(s));
    return SUCCESS;
}
