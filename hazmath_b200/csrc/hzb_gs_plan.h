// hzb_gs_plan.h -- how a Gauss-Seidel schedule is streamed (hzb_gs.cu): the
// layout of its sets and the choice of stages and ring.  Plain C++, so that the
// choice can be checked without a device.
#pragma once
#include <algorithm>
#include <vector>

#ifdef __CUDACC__
#define HZB_HD __host__ __device__
#else
#define HZB_HD
struct int4 { int x, y, z, w; };
#endif

namespace hzb {

// What a CTA holds bounds a schedule that streams: GS_TURNS parts of GS_ROWS
// threads, a row each, and the copying warp (beyond, the row kernels: 670 us a
// sweep of 255^2 points where the stream takes 117), and 16 bytes of shared
// memory a set.
constexpr int GS_ROWS = 256;           // a set's rows: one per computing thread
constexpr int GS_TURNS = 3;            // parts of a CTA that take sets in turn
constexpr int GS_SETS = 2048;          // sets of a schedule (their sizes lie in shared memory)
constexpr int GS_BLOCK = 256;          // places per copy of x
constexpr int GS_PAD = 8;              // set starts and slot pitches, in places
constexpr size_t GS_SMEM = 220 * 1024;

// set s: first place (x), rows and entries per row (y; the latter even and in
// the upper half), the first place's place in the ring (z), first entry (w); its
// rows are rounded up to GS_PAD
HZB_HD inline int gs_pitch(int rows) { return (rows + GS_PAD - 1) / GS_PAD * GS_PAD; }
HZB_HD inline int gs_rows(int4 I) { return I.y & 0xffff; }
HZB_HD inline int gs_width(int4 I) { return I.y >> 16; }
// the places and entries behind a set
HZB_HD inline int gs_end_place(int4 I) { return I.x + gs_pitch(gs_rows(I)); }
HZB_HD inline int gs_end_entry(int4 I) { return I.w + gs_width(I) * gs_pitch(gs_rows(I)); }

// one stage, a group of sets of E entries and R places: values, (b, d), columns
HZB_HD inline size_t gs_stage(int E, int R) {
    return (size_t)E * 8 + (size_t)R * 16 + (size_t)E * 2;
}
inline size_t gs_smem(int ns, int E, int R, int ring, int stages) {
    return (size_t)ns * 16 + (size_t)(ring + 2) * 8 + (size_t)stages * gs_stage(E, R) +
           (size_t)stages * 16;
}

// stages 0: no stream.  uniform: every set's width (0: its own).
struct GsPlan {
    int uniform = 0, group = 0, stages = 0, E = 0, R = 0, ring = 0;
    long long ents = 0;
    std::vector<int4> info;
};

// The plan with one width for all sets, or each set its own; ptr: the sets'
// rows (ns + 1), start: their first places, width: their longest rows (even),
// dist: the largest distance in places between a row and one of its columns.
inline GsPlan gs_plan_width(const std::vector<int> &ptr, const std::vector<int> &start, int places,
                            const std::vector<int> &width, int dist, int uniform) {
    GsPlan P;
    const int ns = (int)ptr.size() - 1;
    P.uniform = uniform;
    P.info.resize(ns);
    for (int k = 0; k < ns; ++k) {
        const int m = ptr[k + 1] - ptr[k], w = uniform ? uniform : width[k];
        if (P.ents > (1LL << 30) || w > 0x7fff) return P;
        P.info[k] = int4{start[k], m | w << 16, 0, (int)P.ents};
        P.ents += (long long)w * gs_pitch(m);
    }
    // Sets per stage and stages: large groups keep the copying warp ahead (it
    // takes about 1 us a group), and the sets in flight have to cover the
    // copies' latency (2 us, ten sets); the first choice that fits.  The ring
    // spans the columns on both sides of the sets in flight.
    //   With one width GS_TURNS parts take the sets in turn, and a part fetches
    // set s when the sets up to s - GS_TURNS are complete.  It waits for a
    // stage's copy by the parity of its round, which only tells neighbouring
    // rounds apart: the round before has to be over by then, that is the group
    // that was in this stage has to lie GS_TURNS sets back.  Stages of fewer
    // than GS_TURNS sets together are for the single sequence only.
    static const int choice[][2] = {{8, 3}, {4, 4}, {4, 3}, {2, 6}, {2, 4}, {1, 8}, {1, 4}, {1, 3}, {1, 2}};
    for (const auto &c : choice) {
        if (uniform && c[0] * c[1] < GS_TURNS) continue;
        P.E = P.R = 0;
        for (int k = 0; k < ns; k += c[0]) {
            const int l = std::min(k + c[0], ns) - 1;
            P.E = std::max(P.E, gs_end_entry(P.info[l]) - P.info[k].w);
            P.R = std::max(P.R, gs_end_place(P.info[l]) - P.info[k].x);
        }
        const long long span = 2LL * dist + (long long)(c[1] + 1) * P.R + 2 * GS_BLOCK;
        P.ring = (int)((std::min<long long>(span, places) + GS_BLOCK - 1) / GS_BLOCK * GS_BLOCK);
        if (P.ring > 0xff00 || gs_smem(ns, P.E, P.R, P.ring, c[1]) > GS_SMEM) continue;
        P.group = c[0];
        P.stages = c[1];
        for (auto &I : P.info) I.z = I.x % P.ring;
        break;
    }
    return P;
}

inline GsPlan gs_plan(const std::vector<int> &ptr, const std::vector<int> &start, int places,
                      const std::vector<int> &width, int dist) {
    // Rows of up to 8 entries: one width for all sets, so that the next set's
    // loads need no branch and run ahead of the barrier (0.35 us a set of a 2D
    // level with each set its own width, 0.18 to 0.23 with the longest row's).
    const int longest = *std::max_element(width.begin(), width.end());
    if (longest <= 8) {
        GsPlan P = gs_plan_width(ptr, start, places, width, dist, std::max(2, longest));
        if (P.stages) return P;
    }
    return gs_plan_width(ptr, start, places, width, dist, 0);
}

// Places of the sets (starts rounded to GS_PAD, the end to GS_BLOCK); 0: a set
// has more than a row per thread, or there are too many sets.
inline int gs_places(const std::vector<int> &ptr, std::vector<int> *start) {
    const int ns = (int)ptr.size() - 1;
    if (ns < 1 || ns > GS_SETS) return 0;
    start->resize(ns);
    int places = 0;
    for (int k = 0; k < ns; ++k) {
        const int m = ptr[k + 1] - ptr[k];
        if (m > GS_ROWS) return 0;
        (*start)[k] = places;
        places += gs_pitch(m);
    }
    return (places + GS_BLOCK - 1) / GS_BLOCK * GS_BLOCK;
}

}  // namespace hzb
