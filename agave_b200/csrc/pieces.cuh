// The sequences of a step cut into pieces of `len` tokens, numbered through, sequence by sequence.
#pragma once
#include "common.cuh"

namespace {

struct Piece {
    int seq, part, parts;      // the sequence, the piece's number in it and how many it has
};

// Piece z; false: there is none.  A whole warp calls it (any warp, all with the same z): a lane has
// a sequence, so a batch of 32 is one trip to memory; one thread after another's length took 0.3 us
// a sequence and CTA, which was most of a launch over 256 sequences.
__device__ __forceinline__ bool piece_of(const int* __restrict__ cu, int n_seq, int len, int z, Piece& out) {
    const int lane = threadIdx.x & 31;
    int before = 0;
    for (int e0 = 0; e0 < n_seq; e0 += 32) {
        const int e = e0 + lane;
        const int own = e < n_seq ? (cu[e + 1] - cu[e] + len - 1) / len : 0;
        int upto = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned past = __ballot_sync(0xffffffffu, before + upto > z);
        if (past) {
            const int l = __ffs(past) - 1;
            out.seq = e0 + l;
            out.parts = __shfl_sync(0xffffffffu, own, l);
            out.part = z - (before + __shfl_sync(0xffffffffu, upto, l) - out.parts);
            return true;
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    return false;
}

// The number of sequence seq's first piece.  A whole warp calls it.
__device__ __forceinline__ int first_piece(const int* __restrict__ cu, int seq, int len) {
    const int lane = threadIdx.x & 31;
    int n = 0;
    for (int e = lane; e < seq; e += 32) n += (cu[e + 1] - cu[e] + len - 1) / len;
    return __reduce_add_sync(0xffffffffu, n);
}

}  // namespace
