// Radix selection over the 32-bit keys of a row by the threads of a CTA or of a cluster, whose
// sums are counts or 64-bit fixed point, so that the result does not depend on the order in which
// threads add.
//
// The file that includes this one defines SM_THREADS (threads of a CTA, at least SM_BINS),
// cluster_meet() (all threads of the cluster meet) and peer_u64(p, r) (what CTA r of the cluster
// has where this CTA has p).
#pragma once

constexpr int SM_BINS = 256;
constexpr int SM_PIECE = 14;                   // bits of a fixed-point weight added at a time
constexpr int SM_FOLD = 1 << 18;               // values between two folds: SM_PIECE + 18 <= 32 bits

struct RadixShared {
    unsigned long long mass[2][SM_BINS];       // this slice's bins, read by the whole cluster
    unsigned long long sums[SM_BINS];          // the cluster's
    unsigned part[3][SM_BINS];                 // (counts in part[0]; the pieces of 64-bit sums)
    unsigned prefix;
    unsigned long long above;
};

// The bin in which a sum over the bins from the greatest downwards, starting at `above`, first
// reaches `target` (bin 0 if none does), and the sum over the bins above it.  A warp: lane l has
// bins 8 l .. 8 l + 7 of the cluster's sums.
__device__ __forceinline__ void pick_bin(const unsigned long long (&m)[8], unsigned long long above,
                                         unsigned long long target, int& bin,
                                         unsigned long long& sum_above) {
    const int lane = threadIdx.x & 31;
    unsigned long long own = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) own += m[i];
    unsigned long long tail = own;               // of this lane and the ones above it
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_down_sync(0xffffffffu, tail, o);
        if (lane + o < 32) tail += t;
    }
    unsigned long long acc = above + (tail - own);
    int mine = -1;
    unsigned long long before = 0;
#pragma unroll
    for (int i = 7; i >= 0; --i) {
        if (mine < 0 && acc + m[i] >= target) { mine = lane * 8 + i; before = acc; }
        acc += m[i];
    }
    // (acc: with every bin of the lane; lane 0 stops at bin 0 whatever the sum)
    if (lane == 0 && mine < 0) { mine = 0; before = acc - m[0]; }
    const unsigned have = __ballot_sync(0xffffffffu, mine >= 0);
    const int at = 31 - __clz(have);
    bin = __shfl_sync(0xffffffffu, mine, at);
    sum_above = __shfl_sync(0xffffffffu, before, at);
}

// Descends the 32-bit key space 8 bits at a time, over the whole row (C > 1) or this CTA's slice
// (C = 1).  COUNT: the key of the element at which the count from above reaches target.
// Otherwise the greatest key whose tail mass reaches target (each element weighs its fixed-point
// weight).  each(e0, e1, f): calls f(key, weight) for the thread's elements e0 .. e1 - 1 of at most
// thread_elements.  Every thread calls it; `turn` counts the passes of the kernel, whose two sets of bins
// alternate, so one meeting of the cluster a pass suffices: a set is cleared after the meeting
// of the pass before, when every peer has read it.
template <bool COUNT, typename EachFn>
__device__ unsigned radix_descend(RadixShared& sh, int C, int& turn, unsigned long long target,
                                  int thread_elements, EachFn each) {
    __syncthreads();                       // (everybody has the result of the descent before)
    if (threadIdx.x == 0) { sh.prefix = 0; sh.above = 0; }
    for (int pass = 0; pass < 4; ++pass, ++turn) {
        const int shift = 24 - 8 * pass;
        unsigned long long* bins = sh.mass[turn & 1];
        if (threadIdx.x < SM_BINS) {
            bins[threadIdx.x] = 0;
            sh.part[0][threadIdx.x] = sh.part[1][threadIdx.x] = sh.part[2][threadIdx.x] = 0;
        }
        __syncthreads();
        const unsigned prefix = sh.prefix;
        const unsigned himask = pass == 0 ? 0u : (0xffffffffu << (shift + 8));
        auto fold = [&]() {
            __syncthreads();
            if (threadIdx.x < SM_BINS) {
                const int b = threadIdx.x;
                bins[b] += (unsigned long long)sh.part[0][b] +
                           (COUNT ? 0ull : ((unsigned long long)sh.part[1][b] << SM_PIECE) +
                                           ((unsigned long long)sh.part[2][b] << (2 * SM_PIECE)));
                sh.part[0][b] = sh.part[1][b] = sh.part[2][b] = 0;
            }
            __syncthreads();
        };
        // (a CTA adds SM_FOLD values at most before a fold)
        constexpr int PER = SM_FOLD / SM_THREADS;
        for (int e0 = 0; e0 < thread_elements; e0 += PER) {
            each(e0, min(e0 + PER, thread_elements), [&](unsigned key, unsigned long long m) {
                if ((key & himask) != prefix || m == 0) return;
                const int b = (key >> shift) & 255u;
                if (COUNT) {
                    atomicAdd(&sh.part[0][b], 1u);
                } else if (m >> (3 * SM_PIECE)) {              // (no weight is above 2^40; a NaN's)
                    atomicAdd(&bins[b], m);
                } else {
                    const unsigned lo = (1u << SM_PIECE) - 1;
                    const unsigned p0 = (unsigned)m & lo, p1 = (unsigned)(m >> SM_PIECE) & lo,
                                   p2 = (unsigned)(m >> (2 * SM_PIECE));
                    if (p0) atomicAdd(&sh.part[0][b], p0);
                    if (p1) atomicAdd(&sh.part[1][b], p1);
                    if (p2) atomicAdd(&sh.part[2][b], p2);
                }
            });
            fold();
        }
        if (C > 1) {
            // the cluster's sums: a thread a bin, its peers' loads in flight together
            cluster_meet();
            if (threadIdx.x < SM_BINS) {
                unsigned long long v[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) v[r] = r < C ? peer_u64(&bins[threadIdx.x], r) : 0ull;
                unsigned long long m = 0;
#pragma unroll
                for (int r = 0; r < 8; ++r) m += v[r];
                sh.sums[threadIdx.x] = m;
            }
            __syncthreads();
        }
        if (threadIdx.x < 32) {
            const unsigned long long* of = C > 1 ? sh.sums : bins;
            unsigned long long m[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) m[i] = of[threadIdx.x * 8 + i];
            int bin;
            unsigned long long above;
            pick_bin(m, sh.above, target, bin, above);
            __syncwarp();
            if (threadIdx.x == 0) {
                sh.above = above;
                sh.prefix = prefix | ((unsigned)bin << shift);
            }
        }
        __syncthreads();
    }
    return sh.prefix;
}
