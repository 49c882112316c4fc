// Choosing the next token on the device: arg max, and temperature / top-k /
// top-p sampling; plus the repeat penalty.  A sequence's row of logits (32-bit) is the work
// of several CTAs: slices for the arg max, a cluster's shared memory for sampling.
//
// Reference (src/ops/math.zig): arg max takes the first index on ties (32-50);
// sampling divides by the temperature, keeps values >= the k-th greatest,
// forms exp(x - max), keeps weights >= the weight at which the descending
// running sum first reaches top_p * total, and draws by a linear scan of the
// running sum in index order, falling back to the last index (209-371); the
// repeat penalty divides positive logits and multiplies the others, once per
// occurrence (186-197).
//
// Sums that decide something (the top-p cut and the draw) are kept in 64-bit
// fixed point, so the same seed gives the same token whatever the order in
// which threads add.  The uniform number comes from a hash of (seed, sequence
// id, step): a sequence's draws do not depend on its batch.
#include "common.cuh"

constexpr int SM_THREADS = 1024;
// Sampling options as words on the device, so that one recorded decode step serves
// every setting: [1 / temperature (float bits), top_k, top_p (float bits), seed low,
// seed high, repeat penalty (float bits)]; two spare words.
enum { SP_INV_TEMPERATURE = 0, SP_TOP_K, SP_TOP_P, SP_SEED_LO, SP_SEED_HI, SP_PENALTY, SP_WORDS = 8 };
constexpr double FIX_ONE = 1099511627776.0;    // 2^40

// ----------------------------------------------------------------- arg max
// Two stages so that a few rows still fill the GPU: AM_PARTS CTAs per row each
// find (greatest value, first index) over a slice, the CTA that finishes last for
// a row reduces the slices.  Ties go to the lowest index in both stages.
constexpr int AM_PARTS = 64;
constexpr int AM_THREADS = 256;
constexpr int AM_MAX_ROWS = 4096;
__device__ float g_am_val[AM_MAX_ROWS * AM_PARTS];
__device__ int g_am_idx[AM_MAX_ROWS * AM_PARTS];
__device__ int g_am_count[AM_MAX_ROWS];       // zero between launches

__device__ __forceinline__ void am_better(float& best, int& idx, float ov, int oi) {
    if (ov > best || (ov == best && oi < idx)) { best = ov; idx = oi; }
}

__global__ void __launch_bounds__(AM_THREADS)
argmax_kernel(const float* __restrict__ logits, long long row_stride, int V, int* __restrict__ out,
              int row0) {
    pdl_wait();
    pdl_launch_next();
    __shared__ float sv[32];
    __shared__ int si[32];
    __shared__ int s_last;
    const int row = blockIdx.y, part = blockIdx.x;
    const float* src = logits + (size_t)(row0 + row) * row_stride;
    const int per = (V + AM_PARTS - 1) / AM_PARTS;
    const int lo = part * per, hi = min(V, lo + per);
    float best = -INFINITY;
    int idx = 0x7fffffff;
    for (int i = lo + threadIdx.x; i < hi; i += AM_THREADS) am_better(best, idx, src[i], i);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        am_better(best, idx, __shfl_xor_sync(0xffffffffu, best, o),
                  __shfl_xor_sync(0xffffffffu, idx, o));
    if (lane == 0) { sv[warp] = best; si[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        best = lane < AM_THREADS / 32 ? sv[lane] : -INFINITY;
        idx = lane < AM_THREADS / 32 ? si[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            am_better(best, idx, __shfl_xor_sync(0xffffffffu, best, o),
                      __shfl_xor_sync(0xffffffffu, idx, o));
        if (lane == 0) {
            g_am_val[row * AM_PARTS + part] = best;
            g_am_idx[row * AM_PARTS + part] = idx;
            __threadfence();
            s_last = atomicAdd(&g_am_count[row], 1) == AM_PARTS - 1;
        }
    }
    __syncthreads();
    if (!s_last || warp != 0) return;
    __threadfence();
    best = -INFINITY;
    idx = 0x7fffffff;
    for (int i = lane; i < AM_PARTS; i += 32)
        am_better(best, idx, __ldcg(&g_am_val[row * AM_PARTS + i]),
                  __ldcg(&g_am_idx[row * AM_PARTS + i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
        am_better(best, idx, __shfl_xor_sync(0xffffffffu, best, o),
                  __shfl_xor_sync(0xffffffffu, idx, o));
    if (lane == 0) {
        out[row0 + row] = idx == 0x7fffffff ? 0 : idx;
        g_am_count[row] = 0;
    }
}

// out[b] = first index of the greatest logits[b, :].  Calls on different streams
// must not overlap: the stages share one table of partial results.
AGV_API int agv_argmax(const float* logits, long long row_stride, int B, int V, int* out,
                       cudaStream_t stream) {
    AGV_REQUIRE(B >= 0 && V > 0 && row_stride >= V, "argmax: bad sizes B=%d V=%d", B, V);
    for (int row0 = 0; row0 < B; row0 += AM_MAX_ROWS) {
        const int rows = B - row0 < AM_MAX_ROWS ? B - row0 : AM_MAX_ROWS;
        agv_launch(argmax_kernel, dim3(AM_PARTS, rows), AM_THREADS, 0, stream, logits, row_stride, V, out,
                                                                      row0);
        AGV_LAUNCH_OK("argmax_kernel");
    }
    return 0;
}

// ------------------------------------------------------------ repeat penalty
// Generated ids are kept per cache slot on the device: hist [n_slots, cap] and
// hist_len [n_slots].  A decode step appends its input token (the token chosen
// in the step before), so at any step the history is "everything generated so
// far", which is what the reference penalises (src/main.zig:2350-2352).
__global__ void history_append_kernel(const int* __restrict__ tokens, const int* __restrict__ slots,
                                      int* __restrict__ hist, int* __restrict__ hist_len, int cap,
                                      int B) {
    pdl_wait();
    pdl_launch_next();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B) return;
    const int slot = slots[b];
    if (slot < 0) return;
    const int n = hist_len[slot];
    if (n < cap) {
        hist[(size_t)slot * cap + n] = tokens[b];
        hist_len[slot] = n + 1;
    }
}

AGV_API int agv_history_append(const int* tokens, const int* slots, int* hist, int* hist_len,
                               int cap, int B, cudaStream_t stream) {
    AGV_REQUIRE(cap > 0 && B >= 0, "history_append: bad sizes");
    if (B == 0) return 0;
    agv_launch(history_append_kernel, (B + 127) / 128, 128, 0, stream, tokens, slots, hist, hist_len, cap, B);
    AGV_LAUNCH_OK("history_append_kernel");
    return 0;
}

// A decode step launched before the host has read the step before it takes its
// input tokens from that step's choices on the device: tokens[b] = prev[b] when
// *take is set (ids outside the vocabulary, possible only in padding rows, become 0).
__global__ void take_tokens_kernel(int* __restrict__ tokens, const int* __restrict__ prev,
                                   const int* __restrict__ take, int B, int V) {
    pdl_wait();
    pdl_launch_next();
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= B || !*take) return;
    const int t = prev[b];
    tokens[b] = (t >= 0 && t < V) ? t : 0;
}

AGV_API int agv_take_tokens(int* tokens, const int* prev, const int* take, int B, int V,
                            cudaStream_t stream) {
    AGV_REQUIRE(B >= 0 && V > 0, "take_tokens: bad sizes");
    if (B == 0) return 0;
    agv_launch(take_tokens_kernel, (B + 127) / 128, 128, 0, stream, tokens, prev, take, B, V);
    AGV_LAUNCH_OK("take_tokens_kernel");
    return 0;
}

// The thread of an id's first occurrence applies the penalty once per
// occurrence, so no two threads touch one logit.
__global__ void repeat_penalty_kernel(float* __restrict__ logits, long long row_stride, int V,
                                      const int* __restrict__ slots, const int* __restrict__ hist,
                                      const int* __restrict__ hist_len, int cap, float penalty,
                                      const int* __restrict__ dev_params) {
    pdl_wait();
    pdl_launch_next();
    if (dev_params) penalty = __int_as_float(dev_params[SP_PENALTY]);
    if (penalty == 1.0f) return;
    const int b = blockIdx.y;
    const int slot = slots[b];
    if (slot < 0) return;
    const int n = min(hist_len[slot], cap);
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int* hrow = hist + (size_t)slot * cap;
    const int id = hrow[i];
    if (id < 0 || id >= V) return;
    int count = 0;
    for (int j = 0; j < n; ++j) {
        if (hrow[j] == id) {
            if (j < i) return;
            ++count;
        }
    }
    float* p = logits + (size_t)b * row_stride + id;
    float v = *p;
    for (int c = 0; c < count; ++c) v = v > 0.f ? v / penalty : v * penalty;
    *p = v;
}

// logits [B, V] in place; slots [B]; hist [n_slots, cap]; hist_len [n_slots].
// dev_params (or null): the sampling words on the device (see agv_sample); the penalty
// is then read from them when the kernel runs, not from the argument.
AGV_API int agv_repeat_penalty(float* logits, long long row_stride, int B, int V, const int* slots,
                               const int* hist, const int* hist_len, int cap, float penalty,
                               const int* dev_params, cudaStream_t stream) {
    AGV_REQUIRE(dev_params || penalty > 0.f, "repeat_penalty: penalty must be positive");
    AGV_REQUIRE(cap > 0, "repeat_penalty: bad history capacity");
    if (B == 0) return 0;
    dim3 grid((cap + 255) / 256, B);
    agv_launch(repeat_penalty_kernel, grid, 256, 0, stream, logits, row_stride, V, slots, hist, hist_len,
                                                    cap, penalty, dev_params);
    AGV_LAUNCH_OK("repeat_penalty_kernel");
    return 0;
}

// ------------------------------------------------------------------ sampling
__device__ __forceinline__ unsigned ordered_key(float v) {
    const unsigned u = __float_as_uint(v);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ unsigned long long splitmix64(unsigned long long x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}
// A weight in fixed point, cut off.  Weights are at most 1: the 24 bits of the number shifted to
// their place, without the 64-bit conversions, of which an SM makes a sixteenth of what it
// shifts.  (An infinity or a NaN goes by them.)
__device__ __forceinline__ unsigned long long to_fixed(float w) {
    const unsigned u = __float_as_uint(w);
    const int e = (int)(u >> 23);                       // (sign clear)
    if (e > 127) return (unsigned long long)((double)w * FIX_ONE);
    const unsigned long long m = (u & 0x7fffffu) | 0x800000u;
    return e >= 110 ? m << (e - 110) : e > 110 - 24 ? m >> (110 - e) : 0ull;
}

// A row is shared by the C CTAs of a cluster (C = 1, 2, 4 or 8): CTA c owns a contiguous slice of
// the vocabulary, keeps it in shared memory (`resident` values at most; what a larger slice has
// beyond them is read again from global memory) and answers for it in every pass.  What decides
// anything crosses the cluster: the maximum, the 256 bins of a radix pass, the slices' sums.
// All of those are maxima, counts and fixed-point sums, so the token does not depend on C.
//
// What bounds it: the passes over the slice and the cluster barriers, not the bytes (64 rows of
// 262,144 logits are 67 MB, 10 us of HBM).  One CTA a row, every pass over the row in L2 and a
// 64-bit shared-memory atomic for every value of a bin, took 4,000 us for those 64 rows alone and
// 6,600 us in a decode step, where the CTAs of the step's next kernel wait on the same SMs.  With
// slices in shared memory, top-k 64 and top-p 0.95: 334 us when every pass runs over the cluster,
// 100 us when the few candidates a top-k leaves are finished by one CTA (one row: 3,860, 72 and 33
// us; top-p 0.9 alone, where every weight takes part: 2,160 -> 326 us).  Eight CTAs of a 262,144
// row take 128 KB each, so 16 to 18 rows run at a time.  CTAS: how many an SM is to hold; two have 32 registers
// a thread, which costs a lone CTA its spills (one row of 65,536, top-k 64 21.9 -> 25.4 us) and gains where
// there are more than SMs and their slices leave room (256 rows of 20,000, temperature alone 42 -> 30).
constexpr int SM_RESIDENT = 44 * 1024;         // values of a slice in shared memory (176 KB)
constexpr int SM_LIST = 2048;                  // candidates of a top-k that one CTA finishes alone

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// All threads of the cluster meet, and see what the others wrote before.
__device__ __forceinline__ void cluster_meet() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;"
                 ::: "memory");
}
__device__ __forceinline__ unsigned peer_address(const void* mine, int rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(mine)), "r"(rank));
    return a;
}
__device__ __forceinline__ unsigned long long peer_u64(const unsigned long long* mine, int rank) {
    unsigned long long v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(peer_address(mine, rank)) : "memory");
    return v;
}
__device__ __forceinline__ unsigned peer_u32(const void* mine, int rank) {
    unsigned v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(peer_address(mine, rank)) : "memory");
    return v;
}
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

#include "radix.cuh"

struct SampleShared : RadixShared {
    unsigned long long wsum[SM_THREADS / 32];  // kept weight of every warp's range
    unsigned long long slice_sum;              // read by the whole cluster
    unsigned long long total_mass;             // read by the whole cluster
    float red[32];
    float mx;                                  // read by the whole cluster
    unsigned bound;                            // read by the whole cluster
    int n_list;                                // read by the whole cluster
    float list_x[SM_LIST];                     // CTA 0's: written by the whole cluster
    int list_i[SM_LIST];
};

template <int CTAS>
__global__ void __launch_bounds__(SM_THREADS, CTAS)
sample_kernel(const float* __restrict__ logits, long long row_stride, int V, int C, int slice, int resident,
              int* __restrict__ out, float inv_temperature, int top_k, float top_p,
              unsigned long long seed, const long long* __restrict__ seq_ids,
              const int* __restrict__ steps, const int* __restrict__ dev_params) {
    pdl_wait();
    pdl_launch_next();
    if (dev_params) {
        inv_temperature = __int_as_float(dev_params[SP_INV_TEMPERATURE]);
        top_k = dev_params[SP_TOP_K];
        top_p = __int_as_float(dev_params[SP_TOP_P]);
        seed = (unsigned long long)(unsigned)dev_params[SP_SEED_LO] |
               ((unsigned long long)(unsigned)dev_params[SP_SEED_HI] << 32);
    }
    __shared__ SampleShared sh;
    extern __shared__ __align__(16) float sm_slice[];
    float* val = sm_slice;                                // the slice: logits, then weights
    bool listed = false;                                  // the candidates instead of the slice
    const int rank = C > 1 ? (int)cluster_rank() : 0;
    const int row_id = blockIdx.x / C;
    const float* row = logits + (size_t)row_id * row_stride;
    const int lo = min(V, rank * slice);
    int n = min(V, lo + slice) - lo;
    int held = min(n, resident);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int elements = (n + SM_THREADS - 1) / SM_THREADS;            // of a thread, SM_THREADS apart
    int turn = 0;

    // 1. the slice, divided by the temperature; its maximum and the thread's greatest key
    float mx = -INFINITY;
    unsigned best = 0;
    auto take = [&](int i, float raw) {
        const float x = raw * inv_temperature;
        mx = fmaxf(mx, x);
        best = max(best, ordered_key(x));
        if (i < resident) val[i] = x;
    };
    if (((uintptr_t)(row + lo) & 15) == 0) {
        const float4* src = reinterpret_cast<const float4*>(row + lo);
#pragma unroll 4
        for (int i = tid; i < n / 4; i += SM_THREADS) {
            const float4 v = __ldcs(src + i);
            take(4 * i, v.x); take(4 * i + 1, v.y); take(4 * i + 2, v.z); take(4 * i + 3, v.w);
        }
        for (int i = n / 4 * 4 + tid; i < n; i += SM_THREADS) take(i, row[lo + i]);
    } else {
#pragma unroll 4
        for (int i = tid; i < n; i += SM_THREADS) take(i, row[lo + i]);
    }
    mx = block_max(mx, sh.red);
    auto scaled = [&](int i) { return i < held ? val[i] : row[lo + i] * inv_temperature; };

    // 2. top-k threshold on the scaled logits.  The k-th greatest of the threads' greatest keys
    // is at most the k-th greatest key of the slice, and that at most the row's: only elements
    // that reach the best such bound of the cluster are counted.
    const bool by_count = top_k > 0 && top_k < V;
    unsigned bound = 0;
    if (by_count && top_k <= SM_THREADS) {
        bound = radix_descend<true>(sh, 1, turn, (unsigned long long)top_k, 1,
                                    [&](int, int, auto&& add) { add(best, 1ull); });
    }
    if (C > 1) {
        if (tid == 0) { sh.mx = mx; sh.bound = bound; }
        cluster_meet();
        for (int r = 0; r < C; ++r) {
            mx = fmaxf(mx, __uint_as_float(peer_u32(&sh.mx, r)));
            bound = max(bound, peer_u32(&sh.bound, r));
        }
    }
    // Where a top-k left few candidates (about C k of them), CTA 0 gets them all, in index order,
    // and finishes alone: the meetings of the cluster are what the passes below cost.
    auto index_range = [&](int& a, int& b) {              // a warp's, in whole 32s
        const int per = ((n + SM_THREADS / 32 - 1) / (SM_THREADS / 32) + 31) / 32 * 32;
        a = min(n, warp * per);
        b = min(n, a + per);
    };
    if (C > 1 && by_count && top_k <= SM_THREADS) {
        int a, b, count = 0;
        index_range(a, b);
        for (int i = a + lane; i < b; i += 32) count += ordered_key(scaled(i)) >= bound;
        count = __reduce_add_sync(0xffffffffu, count);
        if (lane == 0) sh.wsum[warp] = (unsigned long long)count;
        __syncthreads();
        const int of_warp = (int)sh.wsum[lane];
        const int all = __reduce_add_sync(0xffffffffu, of_warp);
        int at = __reduce_add_sync(0xffffffffu, lane < warp ? of_warp : 0);
        if (tid == 0) sh.n_list = all;
        cluster_meet();
        int total = 0;
        for (int r = 0; r < C; ++r) {
            const int c = (int)peer_u32(&sh.n_list, r);
            if (r < rank) at += c;
            total += c;
        }
        if (total <= SM_LIST) {
            const unsigned px = peer_address(sh.list_x, 0), pi = peer_address(sh.list_i, 0);
            for (int i0 = a; i0 < b; i0 += 32) {
                const int i = i0 + lane;
                const float x = i < b ? scaled(i) : 0.f;
                const bool is = i < b && ordered_key(x) >= bound;
                const unsigned who = __ballot_sync(0xffffffffu, is);
                if (is) {
                    const unsigned o = 4u * (unsigned)(at + __popc(who & ((1u << lane) - 1)));
                    asm volatile("st.shared::cluster.f32 [%0], %1;" :: "r"(px + o), "f"(x) : "memory");
                    asm volatile("st.shared::cluster.u32 [%0], %1;" :: "r"(pi + o), "r"(lo + i) : "memory");
                }
                at += __popc(who);
            }
            cluster_meet();
            if (rank != 0) return;
            listed = true;
            val = sh.list_x;
            n = held = total;
            elements = (n + SM_THREADS - 1) / SM_THREADS;
            bound = 0;
            C = 1;
        }
    }
    unsigned kth_key = 0;
    if (by_count)
        kth_key = radix_descend<true>(sh, C, turn, (unsigned long long)top_k, elements,
                                      [&](int e0, int e1, auto&& add) {
            for (int e = e0; e < e1; ++e) {
                const int i = tid + e * SM_THREADS;
                if (i >= n) break;
                const unsigned key = ordered_key(scaled(i));
                if (key >= bound) add(key, 1ull);
            }
        });
    // 3. the weights take the logits' place; their sum
    auto weigh = [&](float x) { return ordered_key(x) < kth_key ? 0.f : expf(x - mx); };
    for (int i = tid; i < held; i += SM_THREADS) val[i] = weigh(val[i]);
    auto weight = [&](int i) { return i < held ? val[i] : weigh(row[lo + i] * inv_temperature); };
    unsigned cut_bits = 0;
    if (top_p > 0.f && top_p < 1.f) {
        // top-p threshold (the weights are >= 0, so their bits order them)
        unsigned long long part = 0;
        for (int i = tid; i < n; i += SM_THREADS) part += to_fixed(weight(i));
        part = warp_sum_u64(part);
        if (lane == 0) sh.wsum[warp] = part;
        __syncthreads();
        if (warp == 0) {
            part = warp_sum_u64(sh.wsum[lane]);
            if (lane == 0) sh.total_mass = part;
        }
        __syncthreads();
        unsigned long long total = sh.total_mass;
        if (C > 1) {
            cluster_meet();
            total = 0;
            for (int r = 0; r < C; ++r) total += peer_u64(&sh.total_mass, r);
        }
        const unsigned long long target = (unsigned long long)((double)top_p * (double)total);
        cut_bits = radix_descend<false>(sh, C, turn, target > 0 ? target : 1ull, elements,
                                        [&](int e0, int e1, auto&& add) {
            for (int e = e0; e < e1; ++e) {
                const int i = tid + e * SM_THREADS;
                if (i >= n) break;
                const float w = weight(i);
                if (w != 0.f) add(__float_as_uint(w), to_fixed(w));
            }
        });
    }
    __syncthreads();
    auto kept = [&](int i) -> unsigned long long {
        const float w = weight(i);
        return __float_as_uint(w) >= cut_bits ? to_fixed(w) : 0ull;
    };
    // 4. draw in index order: a contiguous range per warp (whole 32s), sums over the ranges
    int w0, w1;
    index_range(w0, w1);
    unsigned long long mine = 0;
    for (int i = w0 + lane; i < w1; i += 32) mine += kept(i);
    mine = warp_sum_u64(mine);
    if (lane == 0) sh.wsum[warp] = mine;
    __syncthreads();
    unsigned long long upto = sh.wsum[lane];               // inclusive sums over the warps
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long t = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += t;
    }
    unsigned long long total = __shfl_sync(0xffffffffu, upto, 31);
    unsigned long long before = __shfl_sync(0xffffffffu, upto, warp) - mine;   // ranges before this warp's
    if (C > 1) {
        if (tid == 0) sh.slice_sum = total;
        cluster_meet();
        total = 0;
        for (int r = 0; r < C; ++r) {
            const unsigned long long s = peer_u64(&sh.slice_sum, r);
            if (r < rank) before += s;
            total += s;
        }
    }
    const unsigned long long h =
        splitmix64(splitmix64(seed ^ 0xA5A5A5A5DEADBEEFull) ^
                   splitmix64((unsigned long long)seq_ids[row_id] * 0x100000001B3ull +
                              (unsigned long long)(unsigned)steps[row_id]));
    const double u = (double)(h >> 11) * (1.0 / 9007199254740992.0);     // [0, 1)
    const unsigned long long thr = (unsigned long long)(u * (double)total);
    if (mine > 0 && before <= thr && thr < before + mine) {
        unsigned long long run = before;
        for (int i0 = w0; i0 < w1; i0 += 32) {
            unsigned long long sum = i0 + lane < w1 ? kept(i0 + lane) : 0ull;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned long long t = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += t;
            }
            const unsigned over = __ballot_sync(0xffffffffu, thr < run + sum);
            if (over) {
                const int i = i0 + __ffs(over) - 1;
                if (lane == 0) out[row_id] = listed ? sh.list_i[i] : lo + i;
                break;
            }
            run += __shfl_sync(0xffffffffu, sum, 31);
        }
    }
    // (no weight at all, or a sum that rounds up to the total: the last index)
    if (rank == 0 && tid == 0 && thr >= total) out[row_id] = V - 1;
    // a CTA's shared memory stays until its peers have read it
    if (C > 1) cluster_meet();
}

// One token per row of logits [B, V].  temperature > 0; top_k 0 = off; top_p
// outside (0, 1) = off.  seq_ids[b] and steps[b] key the draw of row b.
// dev_params (or null): SP_WORDS ints on the device that replace temperature, top_k,
// top_p and seed when the kernel runs (a recorded launch then serves every setting).
AGV_API int agv_sample(const float* logits, long long row_stride, int B, int V, int* out,
                       float temperature, int top_k, float top_p, unsigned long long seed,
                       const long long* seq_ids, const int* steps, const int* dev_params,
                       cudaStream_t stream) {
    AGV_REQUIRE(B >= 0 && V > 0 && row_stride >= V, "sample: bad sizes B=%d V=%d", B, V);
    AGV_REQUIRE(dev_params || temperature > 0.f,
                "sample: temperature must be positive (0 is arg max)");
    AGV_REQUIRE(top_k >= 0, "sample: top_k must be >= 0");
    if (B == 0) return 0;
    // A slice of at most 32,768 values (32 a thread) where eight CTAs can give that; a slice starts
    // on a multiple of four values, so that a row on a 16-byte boundary is read 16 bytes at a time.  Rows for
    // every SM that have only a temperature make no passes over bins: a CTA for up to 40,960 values (256 rows of
    // 40,000: 54 us, 87 with clusters of four).
    const bool plain = !dev_params && top_k == 0 && !(top_p > 0.f && top_p < 1.f) && B > 148;
    int C = 1;
    while (C < 8 && V > (plain ? 40960 : 16384) * C) C *= 2;
    const int slice = ((V + C - 1) / C + 3) / 4 * 4, resident = slice < SM_RESIDENT ? slice : SM_RESIDENT;
    AGV_REQUIRE((long long)B * C <= 0x7fffffffLL, "sample: %d rows exceed the grid limit", B);
    const size_t smem = (size_t)resident * sizeof(float);
    const bool two = (long long)B * C > 148 && 2 * (smem + sizeof(SampleShared) + 1024) <= 227 * 1024;
    auto kern = two ? sample_kernel<2> : sample_kernel<1>;
    AGV_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     SM_RESIDENT * (int)sizeof(float)));
    agv_launch_cluster(kern, dim3((unsigned)(B * C)), SM_THREADS, smem, stream, dim3(C), logits,
                       row_stride, V, C, slice, resident, out, dev_params ? 1.0f : 1.0f / temperature, top_k,
                       top_p, seed, seq_ids, steps, dev_params);
    AGV_LAUNCH_OK("sample_kernel");
    return 0;
}
