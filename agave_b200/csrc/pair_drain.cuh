// The rest of a CTA pair's ring after an abort (plain C++: the host test builds it too).
#pragma once
#ifndef __CUDACC__
#define __device__
#define __forceinline__ inline
#endif

// Both loaders of a pair count a stage's bytes on the even CTA's barrier, which that CTA's loader
// arms for the two of them; after an abort one may have issued stages that the other has not.
// `mine` and `other`: the stages that the even and the odd CTA issued, none of them still issuing.
// Runs in one thread of the even CTA and ends when every copy has landed: a stage that only the odd
// CTA issued is armed for its bytes alone (arm), one that only the even CTA issued gets the bytes
// that nobody will send (fill).  Stages before the ring's last round were consumed, or the loader that
// is ahead would have waited.
template <typename Arm, typename Fill, typename Wait>
__device__ __forceinline__ void pair_drain(int mine, int other, int stages, Arm&& arm, Fill&& fill,
                                           Wait&& wait) {
    const int most = mine > other ? mine : other;
    for (int i = most > stages ? most - stages : 0; i < most; ++i) {
        if (i >= mine) arm(i % stages);
        else if (i >= other) fill(i % stages);
        wait(i % stages, (i / stages) & 1);
    }
}
