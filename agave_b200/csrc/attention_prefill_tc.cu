// Prompt attention on the fifth-generation tensor cores (bfloat16): a flash-style
// kernel over the step's own keys and values, causal with an optional window,
// ragged over the sequences of a batch.
//
// One CTA owns 128 query rows of one sequence: the G query heads that share a
// key/value head times 128 / G consecutive tokens (G = heads per kv head when that
// divides 128 and is at most 16, else one head and 128 tokens), so a key/value tile
// is loaded once for all heads that read it.  Keys come in tiles of 128 positions, two
// halves of 64; a half with no visible key is neither multiplied nor loaded.
//
//   S = Q K^T     tcgen05.mma M 128, N 128, K 16 over head_dim; Q [128 x hd] and
//                 K [128 x hd] are K-major tiles that TMA brings (128-byte swizzle);
//                 S is a 32-bit accumulator in tensor memory, two buffers.
//   softmax       two warpgroups, each with one half of every row's scores (a thread a row,
//                 its TMEM lane): read with tcgen05.ld, bounds applied as a bit a key, running
//                 maximum and sum in 32-bit, the row's maximum exchanged between the two warps
//                 that share it; P rounded to bfloat16 and written over S in tensor memory.
//                 O is only rescaled when the maximum grows by more than 2^8 (the sum carries
//                 the same stale maximum, so the result is the same up to rounding).
//   O += P V      tcgen05.mma M 128, N hd, K 16 over the keys, P from tensor memory; the V
//                 operand must be K-major too, i.e. [hd x keys]: a small kernel first writes
//                 the step's values transposed, each sequence padded to a multiple of
//                 64 columns (zeros), so every half tile starts on a 128-byte boundary.
//
// Warp roles: warp 0 loads queries and keys, warp 3 values (TMA), warp 1 allocates tensor
// memory and issues S = Q K^T, warp 2 issues O += P V, warps 4-11 are the softmax and the
// epilogue.  S of tile j + 1 is computed while the softmax of tile j runs.  Every wait on an
// mbarrier is bounded; when one gives up the kernel records a code, stops, frees its tensor
// memory and returns.
//
// What bounds it: with heads of 128 the exponentials (16,384 a tile at 16 a clock), with heads of
// 256 shared memory (a tile's products read 256 KB of it and TMA writes 128 KB); with few tiles a
// CTA its start and end (4 us).  Against tiles of 64 keys with one softmax warpgroup, P through
// shared memory and rows stored a thread a row (us): one sequence of 2,048, four heads of 256, one kv
// head 43.9 -> 32.7, with a window of 512 21.4 -> 14.7; 4,001 with eight heads of 256 and four kv heads
// 124 -> 90; 2,048 with sixteen heads of 128 76 -> 42, with a bias by distance and a window of
// 1,024 79 -> 46; eight sequences of 256 to 1,024 in blocks 123 -> 72.  One issuing thread for both products was
// slower than the old form with heads of 256 (62 us): it is what such a thread does between two products
// (a wait on a barrier, a commit: 100 to 200 cycles each) that adds up, so slots are large and every
// role has a thread of its own.
//
// Reference: online softmax per (token, head) over KV tiles
// (src/backend/kernels/cuda/sdpa_prefill.zig:26-216); score = (q . k) * scale,
// kv head = h / (nh / nkv) (src/backend/kernels/cpu/sdpa.zig:36-37,58); window
// start sl - W (src/models/gemma4.zig:1153-1155).
#include "common.cuh"
#include "tcgen05.cuh"
#include <map>
#include <tuple>

using namespace tc5;

namespace {

constexpr int AT_M = 128;          // query rows per CTA
constexpr int AT_H = 64;           // keys per half tile
constexpr int AT_N = 2 * AT_H;     // keys per tile
constexpr int AT_THREADS = 384;    // two loaders, two product issuers, two softmax warpgroups
constexpr int AT_SLOT = 32 * 1024; // a slot of the rings of keys and values
constexpr int AT_MAX_SLOTS = 3;    // of each ring
constexpr int AT_O_COL = 2 * AT_N; // tensor memory: two score tiles, then O
constexpr float AT_LAZY = 8.0f;    // log2 units the maximum may lag before O is rescaled

__device__ int g_attn_status = 0;  // 0 ok; else (role << 8) | detail of the first wait that gave up

struct AtArgs {
    __nv_bfloat16* out;            // [T, nh * hdv]
    const int* cu;                 // [B + 1]
    int nh, nkv, hd, G, QT;        // G heads packed per CTA, QT = 128 / G tokens
    int hdv;                       // the value head size (out is [T, nh * hdv])
    int window;
    int keep_first;                // with a window: the first keys that stay visible behind it
    float scale_log2e;
    int kb;                        // 64-element blocks of head_dim
    int k_slots, v_slots;          // slots of the two rings
    int qt_shift;                  // QT is a power of two
    const float* sinks;            // [nh] sink logits joining each row's denominator once, or null
    const float* dist_bias;        // [nh, n_dist] learned bias by distance (unscaled), or null
    int n_dist;
    float inv_scale;               // 1 / scale: the bias joins the raw scores before the scale
    // the soft cap (CAP): a raw score z becomes cap * tanh(z * scale / cap); scale_log2e is then
    // log2(e) alone
    float cap, cap_in;             // cap_in = 2 log2(e) * scale / cap
};

// 2^x by the hardware approximation (relative error about 2^-22; -inf gives 0).
__device__ __forceinline__ float ex2_fast(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Sum of the lengths before sequence b, each rounded up to a multiple of 64.
__device__ __forceinline__ int padded_start(const int* cu, int b) {
    int s = 0;
    for (int i = 0; i < b; ++i) s += (cu[i + 1] - cu[i] + 63) & ~63;
    return s;
}

// ------------------------------------------------------------ V transposed
// vt[(g * hd + d), padded_start(b) + t] = v[cu[b] + t, g, d]; columns between a
// sequence's length and its padded length are zero.
__global__ void __launch_bounds__(256)
transpose_values_kernel(const __nv_bfloat16* __restrict__ v, long long kv_stride,
                        __nv_bfloat16* __restrict__ vt, long long vt_ld,
                        const int* __restrict__ cu, int hd) {
    pdl_wait();
    pdl_launch_next();
    extern __shared__ __nv_bfloat16 tile[];            // [64][hd + 2]
    const int b = blockIdx.z, g = blockIdx.y, t0 = blockIdx.x * 64;
    const int seq0 = cu[b], len = cu[b + 1] - seq0;
    if (t0 >= len) return;
    const int col0 = padded_start(cu, b) + t0;
    const int ld = hd + 2;
    const int pairs = hd / 2;
    for (int i = threadIdx.x; i < 64 * pairs; i += blockDim.x) {
        const int r = i / pairs, c = i % pairs;
        __nv_bfloat162 val = __floats2bfloat162_rn(0.f, 0.f);
        if (t0 + r < len)
            val = *reinterpret_cast<const __nv_bfloat162*>(v + (size_t)(seq0 + t0 + r) * kv_stride +
                                                           (size_t)g * hd + 2 * c);
        *reinterpret_cast<__nv_bfloat162*>(tile + r * ld + 2 * c) = val;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < hd * 32; i += blockDim.x) {
        const int d = i / 32, c = i % 32;               // two tokens per thread
        __nv_bfloat162 val;
        val.x = tile[(2 * c) * ld + d];
        val.y = tile[(2 * c + 1) * ld + d];
        *reinterpret_cast<__nv_bfloat162*>(vt + (size_t)(g * hd + d) * vt_ld + col0 + 2 * c) = val;
    }
}

// ------------------------------------------------------------------ attention
// shared memory beside queries and ring: barriers, the warpgroups' exchange of maxima and sums
constexpr int AT_SMEM_FIXED = 256 + 4 * AT_M * 4;
constexpr int AT_SMEM_MOST = 227 * 1024;

// D[tmem] (+)= A[tmem] B[smem]: A holds 16-bit pairs, 8 columns a step of 16
__device__ __forceinline__ void tc_mma_ts_bf16(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc,
                                               uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// BIAS: the form that adds a table value to every score; CAP: the form with a soft cap on the
// scores (forms of their own, so that the plain form's softmax loop keeps its registers)
template <bool BIAS, bool CAP>
__global__ void __launch_bounds__(AT_THREADS, 1)
attention_prefill_tc_kernel(const __grid_constant__ CUtensorMap map_q,
                            const __grid_constant__ CUtensorMap map_k,
                            const __grid_constant__ CUtensorMap map_vt, AtArgs a) {
    // barriers, tensor memory and the sequence bounds (copied in at the start of the
    // step) are set up while the predecessor still runs; the loader and the softmax
    // warps wait for it before they touch q, k, v or out
    pdl_launch_next();
    extern __shared__ __align__(1024) uint8_t smem[];    // (the swizzle's period)
    const int q_bytes = a.kb * AT_M * 128;              // [kb][128 rows][128 B]
    uint8_t* Qs = smem;
    // Rings of keys and values.  A slot of keys holds up to two 64-element blocks of head_dim
    // ([128 keys][128 B] each); one of values a half tile of up to 256 dims ([dims][64 keys]),
    // or with up to 128 dims both halves.
    uint8_t* Ks = Qs + q_bytes;
    uint8_t* Vs = Ks + a.k_slots * AT_SLOT;
    uint64_t* bars = (uint64_t*)(Vs + a.v_slots * AT_SLOT);
    uint64_t* q_full = bars;                            // [1]
    uint64_t* k_full = bars + 1;                        // [k_slots]
    uint64_t* k_empty = k_full + AT_MAX_SLOTS;
    uint64_t* v_full = k_empty + AT_MAX_SLOTS;          // [v_slots]
    uint64_t* v_empty = v_full + AT_MAX_SLOTS;
    uint64_t* s_full = v_empty + AT_MAX_SLOTS;          // [2]
    uint64_t* p_full = s_full + 2;                      // [2]
    uint64_t* o_done = p_full + 2;                      // [2]
    uint32_t* tmem_slot = (uint32_t*)(o_done + 2);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    float* xmax = (float*)((uint8_t*)bars + 256);       // [2 tiles in turn][2 halves][128 rows]
    static_assert(8 * (1 + 4 * AT_MAX_SLOTS + 6) + 8 <= 256, "barriers must fit their room");

    const int warp = warp_number(), lane = threadIdx.x & 31;
    const int b = blockIdx.z;
    const int seq0 = a.cu[b], len = a.cu[b + 1] - seq0;
    // tiles at the end of a sequence walk the most key tiles: they are scheduled first
    const int q0 = (gridDim.x - 1 - blockIdx.x) * a.QT;
    if (q0 >= len) {
        pdl_wait();
        return;
    }
    const int heads_per_kv = a.nh / a.nkv;
    const int head0 = a.G > 1 ? blockIdx.y * a.G : blockIdx.y;   // first query head of this CTA
    const int kvh = head0 / heads_per_kv;

    // visible key range of this query tile: causal end, window start
    const int j_hi = min(q0 + a.QT - 1, len - 1);
    const int j_lo = first_visible(q0, a.window);
    // the half tiles walked: those of the kept first keys that lie wholly before the window's
    // first, then the window's; two of them make a tile, the last tile may have one only
    const int t_lo = j_lo / AT_H;
    const int n_kept = a.keep_first > 0 ? min((a.keep_first + AT_H - 1) / AT_H, t_lo) : 0;
    const int n_halves = j_hi / AT_H - t_lo + 1 + n_kept;
    const int n_tiles = (n_halves + 1) / 2;
    auto half_of = [&](int i) { return i < n_kept ? i : t_lo + (i - n_kept); };

    if (threadIdx.x == 0) {
        mbar_init(q_full, 1);
        for (int s = 0; s < AT_MAX_SLOTS; ++s) {
            mbar_init(&k_full[s], 1);
            mbar_init(&k_empty[s], 1);
            mbar_init(&v_full[s], 1);
            mbar_init(&v_empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&s_full[s], 1);
            mbar_init(&p_full[s], 8);               // one arrival per softmax warp
            mbar_init(&o_done[s], 1);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    auto give_up = [&](int role, int detail) {
        atomicCAS(&g_attn_status, 0, (role << 8) | detail);
        *abort_flag = 1;
    };

    if (warp == 0) {
        // ------------------------------------------------------------ queries, keys
        if (elect_one()) {
            pdl_wait();
            mbar_expect_tx(q_full, (uint32_t)q_bytes);
            for (int kb = 0; kb < a.kb; ++kb)
                for (int hl = 0; hl < a.G; ++hl)
                    tma_load_3d(Qs + kb * (AT_M * 128) + hl * a.QT * 128, &map_q, kb * 64, head0 + hl,
                                seq0 + q0, q_full);
            int issued = 0, s = 0;
            uint32_t ph = 1;
            for (int j = 0; j < n_tiles && !*abort_flag; ++j) {
                const int y = seq0 + half_of(2 * j) * AT_H;
                const int y2 = 2 * j + 1 < n_halves ? seq0 + half_of(2 * j + 1) * AT_H : -1;
                for (int kb = 0; kb < a.kb; kb += 2) {
                    if (!mbar_wait(&k_empty[s], ph)) {
                        give_up(1, s);
                        break;
                    }
                    const int blocks = min(2, a.kb - kb);
                    uint8_t* d = Ks + s * AT_SLOT;
                    if (a.keep_first) {
                        // the two halves of a tile may lie apart
                        mbar_expect_tx(&k_full[s], (uint32_t)(blocks * (y2 >= 0 ? 2 : 1) * AT_H * 128));
                        for (int i = 0; i < blocks; ++i) {
                            tma_load_3d(d + i * (AT_N * 128), &map_k, (kb + i) * 64, kvh, y, &k_full[s]);
                            if (y2 >= 0)
                                tma_load_3d(d + i * (AT_N * 128) + AT_H * 128, &map_k, (kb + i) * 64, kvh,
                                            y2, &k_full[s]);
                        }
                    } else {
                        // (a last tile of one half brings keys whose scores nobody reads)
                        mbar_expect_tx(&k_full[s], (uint32_t)(blocks * AT_N * 128));
                        for (int i = 0; i < blocks; ++i)
                            tma_load_3d(d + i * (AT_N * 128), &map_k, (kb + i) * 64, kvh, y, &k_full[s]);
                    }
                    ++issued;
                    if (++s == a.k_slots) s = 0, ph ^= 1;
                }
            }
            if (*abort_flag) {
                // wait (bounded) for the copies in flight before the CTA ends
                mbar_wait(q_full, 0);
                for (int i = max(0, issued - a.k_slots); i < issued; ++i)
                    mbar_wait(&k_full[i % a.k_slots], (i / a.k_slots) & 1);
            }
        }
    } else if (warp == 3) {
        // ------------------------------------------------------------ values
        if (elect_one()) {
            const int vt0 = padded_start(a.cu, b);
            pdl_wait();
            int issued = 0, s = 0;
            uint32_t ph = 1;
            const bool apart = a.hdv > 128;                 // a slot a half
            for (int j = 0; j < n_tiles && !*abort_flag; ++j) {
                const int halves = min(2, n_halves - 2 * j);
                for (int h = 0; h < halves; ++h) {
                    if (apart || h == 0) {
                        if (!mbar_wait(&v_empty[s], ph)) {
                            give_up(1, 8 + s);
                            break;
                        }
                        mbar_expect_tx(&v_full[s], (uint32_t)((apart ? 1 : halves) * a.hdv * 128));
                        ++issued;
                    }
                    tma_load_2d(Vs + s * AT_SLOT + (apart ? 0 : h * (AT_SLOT / 2)), &map_vt,
                                vt0 + half_of(2 * j + h) * AT_H, kvh * a.hdv, &v_full[s]);
                    if (apart || h == halves - 1)
                        if (++s == a.v_slots) s = 0, ph ^= 1;
                }
            }
            if (*abort_flag)
                for (int i = max(0, issued - a.v_slots); i < issued; ++i)
                    mbar_wait(&v_full[i % a.v_slots], (i / a.v_slots) & 1);
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------ S = Q K^T
        if (elect_one()) {
            const uint32_t idesc = umma_idesc(AT_M, AT_N);
            const int full_kb = a.hd / 64, tail_steps = (a.hd % 64) / 16;
            const uint64_t q_desc0 = umma_desc(smem_u32(Qs)), k_desc0 = umma_desc(smem_u32(Ks));
            int s = 0;
            uint32_t ph = 0;
            bool ok = mbar_wait(q_full, 0);
            if (!ok) give_up(2, 0);
            for (int j = 0; ok && j < n_tiles && !*abort_flag; ++j) {
                // S of this tile goes where P of the tile before the last one was
                if (j >= 2 && !mbar_wait(&o_done[j & 1], ((j - 2) >> 1) & 1)) {
                    give_up(2, 8 + (j & 1));
                    break;
                }
                const uint32_t d = tmem_base + (j & 1) * AT_N;
                uint64_t qd = q_desc0;
                for (int kb = 0; ok && kb < a.kb; kb += 2) {
                    if (!mbar_wait(&k_full[s], ph)) {
                        give_up(2, 2 + s);
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    uint64_t kd = k_desc0 + (uint64_t)((s * AT_SLOT) >> 4);
                    const int blocks = min(2, a.kb - kb);
                    for (int i = 0; i < blocks; ++i) {
                        const int steps = kb + i < full_kb ? 4 : tail_steps;
#pragma unroll
                        for (int k = 0; k < 4; ++k)
                            if (k < steps)
                                tc_mma_bf16(d, qd + 2 * k, kd + 2 * k, idesc,
                                            (kb + i > 0 || k > 0) ? 1u : 0u);
                        qd += (AT_M * 128) >> 4;
                        kd += (AT_N * 128) >> 4;
                    }
                    tc_commit(&k_empty[s]);
                    if (++s == a.k_slots) s = 0, ph ^= 1;
                }
                if (ok) tc_commit(&s_full[j & 1]);
            }
        }
    } else if (warp == 2) {
        // ------------------------------------------------------------ O += P V
        if (elect_one()) {
            const uint32_t idesc = umma_idesc(AT_M, a.hdv);
            const uint64_t v_desc0 = umma_desc(smem_u32(Vs));
            const bool apart = a.hdv > 128;
            int s = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int j = 0; ok && j < n_tiles && !*abort_flag; ++j) {
                const int halves = min(2, n_halves - 2 * j);
                const uint32_t pa = tmem_base + (j & 1) * AT_N;
                for (int h = 0; h < halves; ++h) {
                    if (apart || h == 0) {
                        if (!mbar_wait(&v_full[s], ph)) {
                            give_up(4, s);
                            ok = false;
                            break;
                        }
                        if (h == 0 && !mbar_wait(&p_full[j & 1], (j >> 1) & 1)) {
                            give_up(4, 8 + (j & 1));
                            ok = false;
                            break;
                        }
                        tc_fence_after();
                    }
                    const uint64_t vd = v_desc0 + (uint64_t)((s * AT_SLOT + (apart ? 0 : h * (AT_SLOT / 2))) >> 4);
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        tc_mma_ts_bf16(tmem_base + AT_O_COL, pa + h * (AT_H / 2) + k * 8, vd + 2 * k, idesc,
                                       (j > 0 || h > 0 || k > 0) ? 1u : 0u);
                    if (apart || h == halves - 1) {
                        tc_commit(&v_empty[s]);
                        if (++s == a.v_slots) s = 0, ph ^= 1;
                    }
                }
                if (ok) tc_commit(&o_done[j & 1]);
            }
        }
    } else if (warp >= 4) {
        // ------------------------------------------------------------ softmax, epilogue
        // Two warpgroups share the rows: each takes one half tile, the row's maximum goes
        // between the two warps of a quarter through shared memory.
        const int wg = (warp >> 2) - 1, quarter = warp & 3;
        const int row = quarter * 32 + lane;                         // TMEM lane = query row
        const int hl = row >> a.qt_shift, tl = row & (a.QT - 1);
        const int qp = q0 + tl;                                       // position in the sequence
        const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const int q_min = q0, q_max = q0 + a.QT - 1;
        // (a barrier of the 64 threads that share these rows)
        auto pair_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(1 + quarter) : "memory"); };
        const int o_half = (a.hdv / 2 + 15) / 16 * 16;                // O's columns are shared too
        const int o_lo = wg ? o_half : 0, o_hi = wg ? a.hdv : o_half;
        float m_used = -INFINITY, l = 0.f;
        // (an answer for the whole warp: what follows is done by all lanes or by none)
        auto wait = [&](uint64_t* bar, uint32_t parity, int detail) -> bool {
            const bool came = __all_sync(0xffffffffu, !*abort_flag && mbar_wait(bar, parity));
            if (!came && lane == 0) give_up(3, detail);
            return came;
        };
        bool ok = true;
        pdl_wait();
        for (int j = 0; j < n_tiles; ++j) {
            const int s = j & 1;
            if (ok) ok = wait(&s_full[s], (j >> 1) & 1, s);
            // (after an abort the warps go on to the barriers of their pairs, without work)
            const bool have = ok && 2 * j + wg < n_halves;
            uint32_t sr[4][16];
            float sv[64];
            float tmax = -INFINITY;
            if (have) {
                tc_fence_after();
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    tc_ld16(lane_addr + s * AT_N + wg * AT_H + c * 16, sr[c]);
                tc_wait_ld();
                if (CAP) {
                    // (before the bounds: a capped -infinity is -cap)
#pragma unroll
                    for (int c = 0; c < 64; ++c) {
                        const float e = ex2_fast(__uint_as_float(sr[c >> 4][c & 15]) * a.cap_in);
                        sr[c >> 4][c & 15] =
                            __float_as_uint(fmaf(__fdividef(2.0f, 1.0f + e), -a.cap, a.cap));
                    }
                }
                const int j0 = half_of(2 * j + wg) * AT_H;
#pragma unroll
                for (int c = 0; c < 64; ++c) sv[c] = __uint_as_float(sr[c >> 4][c & 15]);
                // a half tile every row of the CTA sees whole needs no bounds
                const bool whole = j0 + AT_H - 1 <= q_min &&
                                   (j0 >= first_visible(q_max, a.window) || j0 + AT_H <= a.keep_first);
                if (!whole) {
                    // a bit a key: (behind the window's start, or kept) and not behind the query
                    auto below = [](int n) { return n <= 0 ? 0ull : n >= 64 ? ~0ull : (1ull << n) - 1; };
                    const unsigned long long see =
                        below(qp - j0 + 1) & (~below(first_visible(qp, a.window) - j0) | below(a.keep_first - j0));
                    const unsigned see0 = (unsigned)see, see1 = (unsigned)(see >> 32);
#pragma unroll
                    for (int c = 0; c < 64; ++c)
                        if (!((c < 32 ? see0 : see1) & (1u << (c & 31)))) sv[c] = -INFINITY;
                }
                if (BIAS) {
                    // a learned bias by distance: the last table row stands for all farther keys
                    const float* dbp = a.dist_bias + (size_t)(head0 + hl) * a.n_dist;
                    const int d0 = qp - j0;            // distance of the half tile's first key
                    if (d0 >= 63 && d0 < a.n_dist) {
                        // every key lies behind the query and inside the table: the
                        // row's 64 distances are 64 neighbours of the head's table row
                        const float* dp = dbp + d0;
#pragma unroll
                        for (int c = 0; c < 64; ++c) sv[c] = fmaf(dp[-c], a.inv_scale, sv[c]);
                    } else {
#pragma unroll
                        for (int c = 0; c < 64; ++c) {       // (unrolled whole: sv stays in registers)
                            const int dist = d0 - c;
                            if (dist >= 0)
                                sv[c] = fmaf(dbp[min(dist, a.n_dist - 1)], a.inv_scale, sv[c]);
                        }
                    }
                }
                // the maximum of the raw scores, four chains side by side (the scale is positive)
                float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
                for (int c = 0; c < 64; c += 4) {
                    mx[0] = fmaxf(mx[0], sv[c]);
                    mx[1] = fmaxf(mx[1], sv[c + 1]);
                    mx[2] = fmaxf(mx[2], sv[c + 2]);
                    mx[3] = fmaxf(mx[3], sv[c + 3]);
                }
                tmax = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            }
            // the other half's maximum; behind the barrier both halves' scores have been read,
            // and P may go over them
            float* const xm = xmax + s * 2 * AT_M;
            xm[wg * AT_M + row] = tmax;
            tc_fence_before();
            pair_sync();
            tc_fence_after();
            tmax = fmaxf(tmax, xm[(wg ^ 1) * AT_M + row]) * a.scale_log2e;
            // the maximum in use may lag the true one by up to AT_LAZY
            float factor = 1.f;
            bool rescale = false;
            if (m_used == -INFINITY) {
                m_used = tmax;
            } else if (tmax > m_used + AT_LAZY) {
                factor = exp2f(m_used - tmax);
                m_used = tmax;
                l *= factor;
                rescale = true;
            }
            if (have) {
                const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
                float ps[4] = {0.f, 0.f, 0.f, 0.f};
                uint32_t pk[2][16];
#pragma unroll
                for (int c = 0; c < 64; c += 4) {
                    const float p0 = ex2_fast(fmaf(sv[c], a.scale_log2e, neg_m));
                    const float p1 = ex2_fast(fmaf(sv[c + 1], a.scale_log2e, neg_m));
                    const float p2 = ex2_fast(fmaf(sv[c + 2], a.scale_log2e, neg_m));
                    const float p3 = ex2_fast(fmaf(sv[c + 3], a.scale_log2e, neg_m));
                    ps[0] += p0, ps[1] += p1, ps[2] += p2, ps[3] += p3;
                    const __nv_bfloat162 t0 = __floats2bfloat162_rn(p0, p1);
                    const __nv_bfloat162 t1 = __floats2bfloat162_rn(p2, p3);
                    pk[c >> 5][(c & 31) >> 1] = *reinterpret_cast<const uint32_t*>(&t0);
                    pk[c >> 5][((c & 31) >> 1) + 1] = *reinterpret_cast<const uint32_t*>(&t1);
                }
                l += (ps[0] + ps[1]) + (ps[2] + ps[3]);
                const uint32_t pa = lane_addr + s * AT_N + wg * (AT_H / 2);
                tc_st16(pa, pk[0]);
                tc_st16(pa + 16, pk[1]);
            }
            // O may be rescaled once the product of the last tile ended
            if (ok && __any_sync(0xffffffffu, rescale)) {
                // (the product before that one ended before this tile's scores did)
                ok = wait(&o_done[s ^ 1], ((j - 1) >> 1) & 1, 2);
                if (ok) {
                    tc_fence_after();
                    for (int c = o_lo; c < o_hi; c += 16) {
                        uint32_t o[16];
                        tc_ld16(lane_addr + AT_O_COL + c, o);
                        tc_wait_ld();
#pragma unroll
                        for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
                        tc_st16(lane_addr + AT_O_COL + c, o);
                    }
                }
            }
            tc_wait_st();
            tc_fence_before();
            __syncwarp();
            if (ok && lane == 0) mbar_arrive(&p_full[s]);
        }
        // the row's sum: both halves'
        float* const xl = xmax + (n_tiles & 1) * 2 * AT_M;
        xl[wg * AT_M + row] = l;
        pair_sync();
        l = xl[row] + xl[AT_M + row];                                 // (in one order for both)
        const bool good = ok && wait(&o_done[(n_tiles - 1) & 1], ((n_tiles - 1) >> 1) & 1, 3);
        tc_fence_after();
        if (a.sinks && m_used != -INFINITY)
            l += exp2f(a.sinks[head0 + hl] * 1.4426950408889634f - m_used);
        const float inv = l > 0.f ? 1.0f / l : 0.f;
        // rows leave through shared memory (the rings, used up by now), so that a warp writes
        // whole lines; 16 bytes a row of padding keep both sides free of bank conflicts
        const int ld = a.hdv * 2 + 16;
        uint8_t* const stage = Ks + quarter * 32 * ld;
        if (good)
            for (int c0 = o_lo; c0 < o_hi; c0 += 32) {
                uint32_t o[2][16];
                tc_ld16(lane_addr + AT_O_COL + c0, o[0]);
                if (c0 + 16 < o_hi) tc_ld16(lane_addr + AT_O_COL + c0 + 16, o[1]);
                tc_wait_ld();
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const int c = c0 + q * 16;
                    if (c >= o_hi) break;
                    uint32_t w[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const __nv_bfloat162 t =
                            __floats2bfloat162_rn(__uint_as_float(o[q][2 * i]) * inv,
                                                  __uint_as_float(o[q][2 * i + 1]) * inv);
                        w[i] = *reinterpret_cast<const uint32_t*>(&t);
                    }
                    uint4* d = reinterpret_cast<uint4*>(stage + lane * ld + c * 2);
                    d[0] = make_uint4(w[0], w[1], w[2], w[3]);
                    d[1] = make_uint4(w[4], w[5], w[6], w[7]);
                }
            }
        pair_sync();
        if (good) {
            // 8, 16 or 32 lanes a row
            const int per = a.hdv / 8, sh = per > 16 ? 5 : per > 8 ? 4 : 3;
            const int c = lane & ((1 << sh) - 1);
#pragma unroll 4
            for (int r = (wg << (5 - sh)) + (lane >> sh); r < 32; r += 2 << (5 - sh)) {
                const int rr = quarter * 32 + r, t = rr & (a.QT - 1);
                if (c < per && q0 + t < len)
                    *reinterpret_cast<uint4*>(a.out + (size_t)(seq0 + q0 + t) * ((size_t)a.nh * a.hdv) +
                                              (size_t)(head0 + (rr >> a.qt_shift)) * a.hdv + c * 8) =
                        *reinterpret_cast<const uint4*>(stage + r * ld + c * 16);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                     "r"(512u)
                     : "memory");
    }
}

// A bf16 tensor of up to three dimensions (innermost first), read in boxes with the
// 128-byte swizzle; cached by its geometry.
int make_map_nd(CUtensorMap* out, const void* ptr, int rank, const cuuint64_t* dims,
                const cuuint64_t* strides_bytes, const cuuint32_t* box) {
    typedef std::tuple<const void*, int, unsigned long long, unsigned long long, unsigned long long,
                       unsigned long long, unsigned long long, unsigned, unsigned, unsigned> Key;
    static std::map<Key, CUtensorMap> cache;
    static std::mutex mu;
    Key key(ptr, rank, dims[0], dims[1], rank > 2 ? dims[2] : 0, strides_bytes[0],
            rank > 2 ? strides_bytes[1] : 0, box[0], box[1], rank > 2 ? box[2] : 0);
    {
        std::lock_guard<std::mutex> g(mu);
        auto it = cache.find(key);
        if (it != cache.end()) {
            *out = it->second;
            return 0;
        }
    }
    EncodeTiledFn fn = encode_fn();
    if (!fn) return agv_fail(-4, "attention: the driver does not export cuTensorMapEncodeTiled");
    cuuint32_t estr[3] = {1, 1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(ptr),
                    dims, strides_bytes, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS)
        return agv_fail(-4, "attention: cuTensorMapEncodeTiled failed with code %d", (int)r);
    std::lock_guard<std::mutex> g(mu);
    if (cache.size() > 4096) cache.clear();
    cache[key] = *out;
    return 0;
}

int packed_heads(int nh, int nkv) {
    const int g = nh / nkv;
    return (g > 1 && g <= 16 && 128 % g == 0) ? g : 1;
}

}  // namespace

AGV_API int agv_attention_prefill_tc_supported(int hd, long long q_stride, long long kv_stride) {
    return (hd >= 16 && hd % 16 == 0 && hd <= 256 && q_stride % 8 == 0 && kv_stride % 8 == 0) ? 1 : 0;
}

// Whether a prompt step's attention should take this kernel and not the mma.sync one, where both can:
// T tokens in B sequences of up to max_len; with_vt: the step's q/k/v kernel can write the values
// transposed, else a kernel of its own would.  One CTA of this kernel has the SM, where the other has
// several of 64 rows of one head.  Up to 64 keys that other one walks a single tile, and is ahead where
//  - this kernel needs a second round of the SMs for about as many CTAs as the other has: 16 heads of 64, 16
//    sequences of 12 tokens 9.6 us against 6.1, 64 of 32 tokens 33 against 13; up to twice as many with heads
//    up to 64 (32 over 8, 16 sequences of 64 tokens 9.8 against 8.0); heads of 128 with as many 10.6
//    against 8.3, with twice as many 10.7 against 15.0;
//  - the values would cost a kernel (with the q/k/v kernel: four heads of 256, one kv head, a sequence of 64
//    tokens 19.2 us against 15.0; 16 heads of 64 11.1 against 9.8), but for four and more heads packed into
//    one of so many CTAs (16 over 4 of 128, 64 sequences of 12 tokens 21.7 against 34.1), and for heads
//    that the other one pads (16 heads of 16, 64 tokens 8.8 against 11.2);
//  - sequences have a few tokens each, and their values padded to 64 columns are what takes long: 8 of 4 tokens,
//    16 heads of 64, with the q/k/v kernel 11.4 us against 9.3.
// Everywhere else this kernel is ahead, from one token on: four heads of 256, with the q/k/v kernel 8.2 us
// against 15.2 for 64 tokens, 8.9 against 22.0 for 128.  (1,072 steps of 1 to 4,096 tokens, 16 shapes of
// heads, and 1,134 with ragged ones among them.)
AGV_API int agv_attention_prefill_prefers_tc(int T, int B, int max_len, int nh, int nkv, int hd, int hdv,
                                             int with_vt) {
    const int widest = hd > hdv ? hd : hdv, G = packed_heads(nh, nkv), QT = AT_M / G, sms = 148;
    const long long here = (long long)B * (G > 1 ? nkv : nh) * ((max_len + QT - 1) / QT);
    const long long there = (long long)B * nh * ((max_len + 63) / 64);
    with_vt = with_vt && hd % 64 == 0 && hd == hdv;       // (else the q/k/v kernel calls that of its own)
    // (a few CTAs walking two tiles or three: a kernel for the values takes about what they gain)
    if (max_len > 64) return with_vt || T > 192 || max_len > 128 || widest <= 128;
    if (here > sms && there >= 4 * here) return !with_vt || max_len > 2;
    if (!with_vt) return here <= sms && 8 * widest <= 5 * ((widest + 63) / 64 * 64);
    if (T <= 6LL * B && B >= (widest <= 128 ? 8 : 16)) return 0;
    return here <= sms || there > (widest <= 64 ? 2 : 1) * here;
}

// Columns the transposed-values scratch needs for B sequences of T tokens in all.
AGV_API long long agv_attention_prefill_tc_vt_cols(int T, int B) {
    return ((long long)T + 63LL * B + 63) / 64 * 64;
}


AGV_API int agv_attention_tc_status() {
    int v = 0;
    cudaMemcpyFromSymbol(&v, g_attn_status, sizeof(int));
    if (v) {
        int zero = 0;
        cudaMemcpyToSymbol(g_attn_status, &zero, sizeof(int));
    }
    return v;
}

// vt[(g * hd + d), start(b) + t] = v[cu[b] + t, g, d] for all sequences (start(b):
// the earlier lengths, each rounded up to 64), zeros up to the next multiple of 64.
AGV_API int agv_transpose_values(const void* v, long long kv_stride, void* vt, long long vt_ld,
                                 const int* cu_seqlens, int B, int max_len, int nkv, int hd,
                                 cudaStream_t stream) {
    AGV_REQUIRE(hd % 2 == 0 && kv_stride % 2 == 0 && vt_ld % 2 == 0 && agv_aligned(v, 4) &&
                agv_aligned(vt, 4), "transpose_values: sizes must be even");
    if (B <= 0 || max_len <= 0) return 0;
    dim3 grid((max_len + 63) / 64, nkv, B);
    const size_t smem = (size_t)64 * (hd + 2) * sizeof(__nv_bfloat16);
    agv_launch(transpose_values_kernel, grid, 256, smem, stream, (const __nv_bfloat16*)v, kv_stride,
               (__nv_bfloat16*)vt, vt_ld, cu_seqlens, hd);
    AGV_LAUNCH_OK("transpose_values_kernel");
    return 0;
}

// Whole prompts that start at position 0, bfloat16.  q: [T, nh, hd] rows of
// stride q_stride; k, v: [T, nkv, hd] rows of stride kv_stride; out: [T, nh * hd]
// dense; vt: scratch [nkv * hd, vt_cols] (see agv_attention_prefill_tc_vt_cols);
// cu_seqlens: [B + 1] first token of each sequence; T: rows of q, k and v;
// max_len: the greatest sequence length (sizes the grid).  window 0: no window.
// vt_ready != 0: vt already holds the transposed values (agv_qk_norm_rope_store
// wrote them); else they are transposed here first.
// sinks: [nh] sink logits or null; the scale must be positive.
AGV_API int agv_attention_prefill_tc_ex2(const void* q, long long q_stride, const void* k,
                                         const void* v, long long kv_stride, void* out, void* vt,
                                         long long vt_cols, int vt_ready, const int* cu_seqlens, int B,
                                         int T, int max_len, int nh, int nkv, int hd, float scale,
                                         int window, const float* sinks, const float* dist_bias,
                                         int n_dist, cudaStream_t stream);

AGV_API int agv_attention_prefill_tc_ex3(const void* q, long long q_stride, const void* k,
                                         const void* v, long long kv_stride, void* out, void* vt,
                                         long long vt_cols, int vt_ready, const int* cu_seqlens, int B,
                                         int T, int max_len, int nh, int nkv, int hd, float scale,
                                         int window, const float* sinks, const float* dist_bias,
                                         int n_dist, int keep_first, int hdv, long long v_stride,
                                         float softcap, cudaStream_t stream);

AGV_API int agv_attention_prefill_tc_ex(const void* q, long long q_stride, const void* k,
                                        const void* v, long long kv_stride, void* out, void* vt,
                                        long long vt_cols, int vt_ready, const int* cu_seqlens, int B,
                                        int T, int max_len, int nh, int nkv, int hd, float scale,
                                        int window, const float* sinks, cudaStream_t stream) {
    return agv_attention_prefill_tc_ex2(q, q_stride, k, v, kv_stride, out, vt, vt_cols, vt_ready,
                                        cu_seqlens, B, T, max_len, nh, nkv, hd, scale, window, sinks,
                                        nullptr, 0, stream);
}

// The same with a learned bias by distance: dist_bias [nh, n_dist] is added to the scaled
// score of the key at distance min(t - j, n_dist - 1), or null.
AGV_API int agv_attention_prefill_tc_ex2(const void* q, long long q_stride, const void* k,
                                         const void* v, long long kv_stride, void* out, void* vt,
                                         long long vt_cols, int vt_ready, const int* cu_seqlens, int B,
                                         int T, int max_len, int nh, int nkv, int hd, float scale,
                                         int window, const float* sinks, const float* dist_bias,
                                         int n_dist, cudaStream_t stream) {
    return agv_attention_prefill_tc_ex3(q, q_stride, k, v, kv_stride, out, vt, vt_cols, vt_ready,
                                        cu_seqlens, B, T, max_len, nh, nkv, hd, scale, window, sinks,
                                        dist_bias, n_dist, 0, hd, kv_stride, 0.f, stream);
}

// The same with kept first keys: with a sliding window, position p also sees the keys
// j < keep_first.  hdv, v_stride: the value head size (a multiple of 16 up to 256) and the value
// rows' stride (out is [T, nh * hdv] and vt [nkv * hdv, vt_cols]).  softcap > 0: the scaled score
// s becomes softcap * tanh(s / softcap); not with a distance bias.
AGV_API int agv_attention_prefill_tc_ex3(const void* q, long long q_stride, const void* k,
                                         const void* v, long long kv_stride, void* out, void* vt,
                                         long long vt_cols, int vt_ready, const int* cu_seqlens, int B,
                                         int T, int max_len, int nh, int nkv, int hd, float scale,
                                         int window, const float* sinks, const float* dist_bias,
                                         int n_dist, int keep_first, int hdv, long long v_stride,
                                         float softcap, cudaStream_t stream) {
    AGV_REQUIRE(scale > 0.f, "attention: the tcgen05 kernel takes a positive score scale");
    AGV_REQUIRE(keep_first >= 0 && (keep_first == 0 || window > 0),
                "attention: kept first keys go with a sliding window");
    AGV_REQUIRE(!dist_bias || n_dist > 0, "attention: an empty distance table");
    AGV_REQUIRE(B >= 0 && T >= 0 && nh > 0 && nkv > 0 && hd > 0 && max_len >= 0,
                "attention: bad sizes");
    AGV_REQUIRE(nh % nkv == 0, "attention: %d heads are not a multiple of %d kv heads", nh, nkv);
    AGV_REQUIRE(agv_attention_prefill_tc_supported(hd, q_stride, kv_stride),
                "attention: the tcgen05 kernel needs head_dim (%d) a multiple of 16 up to 256 and "
                "row strides that are multiples of 8", hd);
    AGV_REQUIRE(agv_aligned(q, 16) && agv_aligned(k, 16) && agv_aligned(v, 16) &&
                agv_aligned(out, 16) && agv_aligned(vt, 128),
                "attention: operands must be 16-byte aligned (the scratch 128-byte)");
    AGV_REQUIRE(vt_cols >= agv_attention_prefill_tc_vt_cols(T, B) && vt_cols % 64 == 0,
                "attention: the transposed-values scratch has %lld columns, %lld are needed",
                vt_cols, agv_attention_prefill_tc_vt_cols(T, B));
    AGV_REQUIRE(B <= 65535 && nh <= 65535, "attention: batch or head count exceeds the grid limit");
    AGV_REQUIRE(hdv > 0 && hdv % 16 == 0 && hdv <= 256 && v_stride % 8 == 0,
                "attention: the value head size (%d) must be a multiple of 16 up to 256", hdv);
    AGV_REQUIRE(softcap <= 0.f || !dist_bias, "attention: a soft cap goes without a distance bias");
    if (B == 0 || max_len == 0 || T == 0) return 0;

    AtArgs a;
    a.out = (__nv_bfloat16*)out;
    a.cu = cu_seqlens;
    a.nh = nh, a.nkv = nkv, a.hd = hd, a.hdv = hdv;
    a.G = packed_heads(nh, nkv);
    a.QT = AT_M / a.G;
    a.window = window;
    a.keep_first = keep_first;
    const bool cap = softcap > 0.f;
    a.scale_log2e = (cap ? 1.0f : scale) * 1.4426950408889634f;
    a.cap = softcap;
    a.cap_in = cap ? 2.0f * 1.4426950408889634f * scale / softcap : 0.f;
    a.kb = (hd + 63) / 64;
    a.qt_shift = 0;
    while ((1 << a.qt_shift) < a.QT) ++a.qt_shift;
    // as many slots as fit beside the queries
    int slots = (AT_SMEM_MOST - AT_SMEM_FIXED - a.kb * AT_M * 128) / AT_SLOT;
    if (slots > 2 * AT_MAX_SLOTS) slots = 2 * AT_MAX_SLOTS;
    a.k_slots = (slots + 1) / 2;
    a.v_slots = slots / 2;
    a.sinks = sinks;
    a.dist_bias = dist_bias;
    a.n_dist = n_dist;
    a.inv_scale = 1.0f / scale;

    CUtensorMap mq, mk, mvt;
    {
        cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)nh, (cuuint64_t)T};
        cuuint64_t str[2] = {(cuuint64_t)hd * 2, (cuuint64_t)q_stride * 2};
        cuuint32_t box[3] = {64, 1, (cuuint32_t)a.QT};
        if (int rc = make_map_nd(&mq, q, 3, dims, str, box)) return rc;
    }
    {
        cuuint64_t dims[3] = {(cuuint64_t)hd, (cuuint64_t)nkv, (cuuint64_t)T};
        cuuint64_t str[2] = {(cuuint64_t)hd * 2, (cuuint64_t)kv_stride * 2};
        // (keys a box: half a tile where the halves of a tile may lie apart)
        cuuint32_t box[3] = {64, 1, (cuuint32_t)(keep_first ? AT_H : AT_N)};
        if (int rc = make_map_nd(&mk, k, 3, dims, str, box)) return rc;
    }
    {
        cuuint64_t dims[2] = {(cuuint64_t)vt_cols, (cuuint64_t)nkv * hdv};
        cuuint64_t str[1] = {(cuuint64_t)vt_cols * 2};
        cuuint32_t box[2] = {64, (cuuint32_t)hdv};
        if (int rc = make_map_nd(&mvt, vt, 2, dims, str, box)) return rc;
    }

    if (!vt_ready)
        if (int rc = agv_transpose_values(v, v_stride, vt, vt_cols, cu_seqlens, B, max_len, nkv, hdv,
                                          stream))
            return rc;
    const size_t smem = AT_SMEM_FIXED + (size_t)a.kb * AT_M * 128 + (size_t)slots * AT_SLOT;
    static size_t configured[3] = {0, 0, 0};
    const int form = dist_bias ? 1 : cap ? 2 : 0;
    auto kern = form == 1   ? attention_prefill_tc_kernel<true, false>
                : form == 2 ? attention_prefill_tc_kernel<false, true>
                            : attention_prefill_tc_kernel<false, false>;
    if (smem > configured[form]) {
        AGV_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem));
        configured[form] = smem;
    }
    dim3 grid((max_len + a.QT - 1) / a.QT, a.G > 1 ? nkv : nh, B);
    agv_launch(kern, grid, AT_THREADS, smem, stream, mq, mk, mvt, a);
    AGV_LAUNCH_OK("attention_prefill_tc_kernel");
    return 0;
}

AGV_API int agv_attention_prefill_tc(const void* q, long long q_stride, const void* k,
                                     const void* v, long long kv_stride, void* out, void* vt,
                                     long long vt_cols, int vt_ready, const int* cu_seqlens, int B,
                                     int T, int max_len, int nh, int nkv, int hd, float scale,
                                     int window, cudaStream_t stream) {
    return agv_attention_prefill_tc_ex(q, q_stride, k, v, kv_stride, out, vt, vt_cols, vt_ready,
                                       cu_seqlens, B, T, max_len, nh, nkv, hd, scale, window,
                                       nullptr, stream);
}
