// hzb_tally.h -- the count that the CTAs of a grid take at every crossing of
// their barrier (grid_tally, hzb_kernels.cuh).  Plain C++, so that the protocol
// can be played through without a device.
#pragma once

#ifndef HZB_HD
#ifdef __CUDACC__
#define HZB_HD __host__ __device__
#else
#define HZB_HD
#endif
#endif

namespace hzb {

// Crossing r (1, 2, ..) is taken through word r & 1: arrivals in its lower half,
// what they counted in its upper half, both only ever added to.  A CTA that
// reads the word of crossing r late can find arrivals of crossing r + 1 nowhere
// in it: those go to the other word, and r + 2 has to wait for this CTA.  So
// everyone reads the same count at r, and the total up to r is that plus what
// the other word held when crossing r - 1 was over.  (With one word a late
// reader took counts of r + 1 for r's, and the CTAs could part ways.)
struct GridTally {
    unsigned r = 0;                 // crossings begun
    unsigned before = 0;            // the other word's count, final
    HZB_HD int word() const { return (int)(r & 1u); }
    HZB_HD static unsigned long long arrival(unsigned count) {
        return 1ull | (unsigned long long)count << 32;
    }
    // arrivals that complete the crossing at hand
    HZB_HD bool complete(unsigned long long w, unsigned ctas) const {
        return (int)((unsigned)w - (r + 1u) / 2u * ctas) >= 0;
    }
    HZB_HD unsigned total(unsigned long long w) {
        const unsigned now = (unsigned)(w >> 32), t = now + before;
        before = now;
        return t;
    }
};

}  // namespace hzb
