// Matrix products on the ordinary arithmetic units: out[M, N] = x[M, K] * w[N, K]^T,
// and the gated pair act(x wg^T) * (x wu^T).  This is the whole 32-bit path
// (plain FFMA, no reduced-precision mode) and the fallback of the bfloat16 path
// for shapes the tensor-core kernel refuses.  A plain product may carry the squared relu or the erf GELU.
//
// In 32-bit K (from GS_MIN_K on, rows in whole 16-byte pieces) is cut into eight ranges whose bounds follow from K alone (the last may be short or empty).
// A range is one chain of 32-bit fused multiply-adds in ascending k, and the eight sums are added
// in pairs, ((0+1)+(2+3))+((4+5)+(6+7)), whatever M and N are and however the work is spread: a
// row's result does not depend on which other rows share the launch.
//
// Reference: one dot product per output row, f32 accumulation
// (src/backend/kernels/cuda/gemv_bf16.zig:6-24, gemv_f32.zig:6-21); gated
// activation src/backend/kernels/cuda/gelu_mul.zig:12-19 (here with tanhf).
#include "common.cuh"
#include "act.cuh"

// (the squared relu, max(t, 0)^2, and the erf GELU, t/2 (1 + erf(t / sqrt 2)), go with the
// plain product only)
__device__ __forceinline__ float gelu_tanh_f(float t) {
    const float u = 0.7978845608028654f * (t + 0.044715f * t * t * t);
    return 0.5f * t * (1.0f + tanhf(u));
}
__device__ __forceinline__ float silu_f(float t) { return t / (1.0f + expf(-t)); }
__device__ __forceinline__ float activate(float g, float u, const GateAct& act) {
    if (act.kind == AGV_ACT_CLAMPED) return clamped_gate(g, u, act);
    return (act.kind == AGV_ACT_SILU ? silu_f(g) : gelu_tanh_f(g)) * u;
}

template <bool GATED>
__device__ __forceinline__ float finish(float v, float u, const GateAct& act) {
    if (GATED) return activate(v, u, act);
    if (act.kind == AGV_ACT_RELU2) { v = fmaxf(v, 0.f); return v * v; }
    if (act.kind == AGV_ACT_GELU_ERF) return 0.5f * v * (1.0f + erff(v * 0.7071067811865476f));
    return v;
}

// Any types, alignment and K: tiles of 64 x 64 over all of K, one chain a sum, loads and arithmetic
// in turn.  It stays for bfloat16 data that the tensor-core products refuse and for 32-bit rows that
// are not whole 16-byte pieces, which the other two kernels would have to read a value at a time
// (1152 x 6912, 2,048 rows of bfloat16: 1,340 us here, 2,400 there), and for a K below GS_MIN_K.
constexpr int GA_M = 64, GA_N = 64, GA_K = 16;

template <typename TA, typename TW, typename TO, bool GATED>
__global__ void __launch_bounds__(256)
gemm_any_kernel(const TA* __restrict__ A, const TW* __restrict__ W, const TW* __restrict__ W2,
               TO* __restrict__ C, int M, int N, int K, long long lda, long long ldc, GateAct act) {
    pdl_wait();
    pdl_launch_next();
    __shared__ float As[GA_K][GA_M + 4];
    __shared__ float Ws[GA_K][GA_N + 4];
    __shared__ float Us[GATED ? GA_K : 1][GATED ? GA_N + 4 : 1];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * GA_M, n0 = blockIdx.x * GA_N;
    float acc[4][4] = {};
    float acc2[GATED ? 4 : 1][GATED ? 4 : 1] = {};
    const int lr = tid / 4, lk = (tid % 4) * 4;   // 64 rows x 16 k per tile, 4 k per thread
    for (int k0 = 0; k0 < K; k0 += GA_K) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lk + i;
            const int m = m0 + lr, n = n0 + lr;
            As[lk + i][lr] = (m < M && k < K) ? to_f32(A[(size_t)m * lda + k]) : 0.f;
            Ws[lk + i][lr] = (n < N && k < K) ? to_f32(W[(size_t)n * K + k]) : 0.f;
            if (GATED) Us[lk + i][lr] = (n < N && k < K) ? to_f32(W2[(size_t)n * K + k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GA_K; ++k) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Ws[k][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
            if (GATED) {
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = Us[k][tx * 4 + j];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc2[i][j] = fmaf(a[i], b[j], acc2[i][j]);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + ty * 4 + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= N) continue;
            float v = acc[i][j];
            C[(size_t)m * ldc + n] = from_f32<TO>(finish<GATED>(v, acc2[GATED ? i : 0][GATED ? j : 0], act));
        }
    }
}

// A warp has 32 rows of the weight, one a lane, BM rows of x and R of the eight ranges of K.  The
// weight's pieces of 32 k go through the warp's own ring in shared memory (rows read from global
// memory in whole 128-byte lines, by the lane that owns the row from there); x's pieces are read
// by all lanes at once.  No other warp is waited for until the eight sums are added: the 8 / R
// warps of an output are two a CTA and 4 / R CTAs, a cluster, which read each other's sums.
//
// What bounds it: with few rows of x the weight's bytes, so eight warps share a group of 32
// weight rows where those are few (R = 1: a 1152 x 6912 weight is 36 groups, 288 warps), and a
// warp takes more of K where there are many and the ends of its walk would cost (R = 2, 4); with
// many rows of x the multiply-adds.  3 rows of x, against tiles of 64 x 64 over all of K:
// 1152 x 6912 603 -> 22.4 us, 6912 x 1152 gated 135 -> 26.7, 262144 x 1152 1,284 -> 240 (5.0 TB/s),
// 1536 x 1152 101 -> 12.3 (the figures hold about 6 us of launch and events).
constexpr int GS_ROWS = 32;                    // weight rows of a warp
constexpr int GS_K = 32;                       // k of a piece
constexpr int GS_PITCH = GS_K + 4;             // of a weight row in shared memory (no bank conflict)
constexpr int GS_WARPS = 2;

// Pieces under way a warp (DEEP: see launch_rows).
__host__ __device__ constexpr int gs_stages(int mats, int bm, bool deep) {
    return mats * bm >= 64 ? 3 : deep ? 8 : 4;
}
__host__ __device__ constexpr int gs_stage_floats(int mats, int bm) {
    return mats * GS_ROWS * GS_PITCH + bm * GS_K;
}

// 16 bytes into shared memory, or 16 zero bytes.
__device__ __forceinline__ void gs_copy16(float* dst, const float* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
                 :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// Element (i) of the partial sums that warp `warp` of CTA `rank` of the cluster keeps at `mine`.
__device__ __forceinline__ float gs_peer(const float* mine, int rank) {
    unsigned a;
    float v;
    asm("mapa.shared::cluster.u32 %0, %1, %2;"
        : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(mine)), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}

template <bool GATED, int BM, int R, bool DEEP>
__global__ void __launch_bounds__(GS_WARPS * 32)
gemm_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ W2,
                 float* __restrict__ C, int M, int N, int K, long long lda, long long ldc, GateAct act,
                 int m_tiles, int range) {
    constexpr int MATS = GATED ? 2 : 1, STAGES = gs_stages(MATS, BM, DEEP), CL = 4 / R;
    constexpr int STAGE = gs_stage_floats(MATS, BM), PARTS = 8 / R;
    extern __shared__ __align__(16) float gs_smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = blockIdx.x % CL, tile = blockIdx.x / CL;
    const int n0 = tile / m_tiles * GS_ROWS, m0 = tile % m_tiles * BM;
    float* ring = gs_smem + (size_t)warp * STAGES * STAGE;
    const int r0 = (rank * GS_WARPS + warp) * R;
    const int pieces = (range + GS_K - 1) / GS_K, all = R * pieces;

    const int row = lane >> 3, ch = (lane & 7) * 4;        // of the 16 bytes a lane copies at a time
    // piece t of the walk: its first k and the end of its range
    auto place = [&](int t, int& k0, int& kend) {
        const int r = r0 + (R == 1 ? 0 : t / pieces);
        k0 = r * range + (R == 1 ? t : t % pieces) * GS_K;
        kend = min(K, (r + 1) * range);
    };
    auto fill_w = [&](int t) {
        int k0, kend;
        place(t, k0, kend);
        float* dst = ring + (t % STAGES) * STAGE;
#pragma unroll
        for (int x = 0; x < MATS; ++x, dst += GS_ROWS * GS_PITCH) {
            const float* w = x ? W2 : W;
            const int k = k0 + ch;
#pragma unroll
            for (int i = 0; i < GS_ROWS / 4; ++i) {
                const int n = i * 4 + row;
                const bool there = k < kend && n0 + n < N;
                gs_copy16(dst + n * GS_PITCH + ch, w + (there ? (size_t)(n0 + n) * K + k : 0), there);
            }
        }
    };
    auto fill_x = [&](int t) {
        int k0, kend;
        place(t, k0, kend);
        float* dst = ring + (t % STAGES) * STAGE + MATS * GS_ROWS * GS_PITCH;
        const int k = k0 + ch;
#pragma unroll
        for (int i = 0; i < BM / 4; ++i) {
            const int m = i * 4 + row;
            const bool there = k < kend && m0 + m < M;
            gs_copy16(dst + m * GS_K + ch, A + (there ? (size_t)(m0 + m) * lda + k : 0), there);
        }
    };
    // (the weights are nobody's output: their first pieces are asked for before the wait)
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t)
        if (t < all) fill_w(t);
    pdl_wait();
    pdl_launch_next();
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) {
        if (t < all) fill_x(t);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    float acc[MATS][BM], sum[MATS][BM], high[R == 4 ? MATS : 1][R == 4 ? BM : 1];
#pragma unroll
    for (int x = 0; x < MATS; ++x)
#pragma unroll
        for (int m = 0; m < BM; ++m) acc[x][m] = 0.f;
    int piece = 0, r = 0;
    for (int t = 0; t < all; ++t) {
        asm volatile("cp.async.wait_group %0;" :: "n"(STAGES - 2) : "memory");
        __syncwarp();                          // piece t is there, everybody is past t - 1
        if (t + STAGES - 1 < all) {
            fill_w(t + STAGES - 1);
            fill_x(t + STAGES - 1);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        int k0, kend;
        place(t, k0, kend);
        const float* ws = ring + (t % STAGES) * STAGE + lane * GS_PITCH;
        const float* xs = ring + (t % STAGES) * STAGE + MATS * GS_ROWS * GS_PITCH;
        auto four = [&](int k) {
            const float4 w = *reinterpret_cast<const float4*>(ws + k);
            float4 u;
            if (GATED) u = *reinterpret_cast<const float4*>(ws + GS_ROWS * GS_PITCH + k);
#pragma unroll
            for (int m = 0; m < BM; ++m) {
                const float4 x = *reinterpret_cast<const float4*>(xs + m * GS_K + k);
                float& a = acc[0][m];
                a = fmaf(x.x, w.x, a); a = fmaf(x.y, w.y, a); a = fmaf(x.z, w.z, a); a = fmaf(x.w, w.w, a);
                if (GATED) {
                    float& b = acc[MATS - 1][m];
                    b = fmaf(x.x, u.x, b); b = fmaf(x.y, u.y, b); b = fmaf(x.z, u.z, b); b = fmaf(x.w, u.w, b);
                }
            }
        };
        const int len = kend - k0;
        if (len >= GS_K) {
#pragma unroll
            for (int k = 0; k < GS_K; k += 4) four(k);
        } else {
            for (int k = 0; k < len; k += 4) four(k);
        }
        if (++piece == pieces) {               // the end of a range: its sum takes its place
            piece = 0;
#pragma unroll
            for (int x = 0; x < MATS; ++x)
#pragma unroll
                for (int m = 0; m < BM; ++m) {
                    const float v = acc[x][m];
                    acc[x][m] = 0.f;
                    if (r == 0) sum[x][m] = v;
                    else if (r == 1) sum[x][m] += v;
                    else if constexpr (R == 4) {
                        if (r == 2) high[x][m] = v;
                        else sum[x][m] += high[x][m] + v;
                    }
                }
            ++r;
        }
    }
    // the warps' sums, each in its own ring (its last copies have landed), and the outputs dealt
    // round the threads of the cluster
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int x = 0; x < MATS; ++x)
#pragma unroll
        for (int m = 0; m < BM; ++m) ring[(x * BM + m) * 32 + lane] = sum[x][m];
    if (CL > 1)
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    else
        __syncthreads();
    const int rows = min(BM, M - m0);
    for (int o = rank * GS_WARPS * 32 + threadIdx.x; o < rows * 32; o += CL * GS_WARPS * 32) {
        const int m = o >> 5, n = n0 + (o & 31);
        float v[MATS];
#pragma unroll
        for (int x = 0; x < MATS; ++x) {
            float p[PARTS];
#pragma unroll
            for (int j = 0; j < PARTS; ++j) {
                const float* at = gs_smem + (size_t)(j % GS_WARPS) * STAGES * STAGE + (x * BM + m) * 32 + (o & 31);
                p[j] = CL > 1 ? gs_peer(at, j / GS_WARPS) : *at;
            }
#pragma unroll
            for (int w = 1; w < PARTS; w *= 2)
#pragma unroll
                for (int j = 0; j < PARTS; j += 2 * w) p[j] += p[j + w];
            v[x] = p[0];
        }
        if (n >= N) continue;
        C[(size_t)(m0 + m) * ldc + n] = finish<GATED>(v[0], v[MATS - 1], act);
    }
    if (CL > 1)                                // a CTA's sums stay until its peers have read them
        asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// More than a few rows of x: a CTA has 64 rows of x, 128 outputs a row (64 of each weight in the
// gated form) and one of the eight ranges of K, a thread 8 x 8 sums, so that a 16-byte read of
// shared memory feeds 16 multiply-adds; pieces of 16 k come through a ring of asynchronous copies.
// The eight CTAs of a tile are a cluster: each leaves its sums in shared memory and adds up, in the
// order above, an eighth of the rows.
//
// Bound by the multiply-adds and, beside them, the reads of shared memory.  64 rows against the
// 64 x 64 tiles over all of K: 1152 x 6912 623 -> 76 us, 6912 x 1152 gated 141 -> 80; 2,048 rows: 1,323
// -> 850 (38 TFLOP/s), 2,118 -> 1,813 (36).
constexpr int GT_M = 64, GT_N = 128, GT_K = 16, GT_PITCH = GT_K + 4, GT_STAGES = 4, GT_THREADS = 128;
constexpr int GT_STAGE = (GT_M + GT_N) * GT_PITCH;
static_assert(GT_STAGES * GT_STAGE >= GT_M * GT_N, "the sums take the ring's place");

__device__ __forceinline__ void gt_four(float (&acc)[8][8], const float* xs, const float* ws, int k) {
    float4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = *reinterpret_cast<const float4*>(xs + 8 * i * GT_PITCH + k);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const float4 w = *reinterpret_cast<const float4*>(ws + 16 * j * GT_PITCH + k);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            float& a = acc[i][j];
            a = fmaf(x[i].x, w.x, a); a = fmaf(x[i].y, w.y, a);
            a = fmaf(x[i].z, w.z, a); a = fmaf(x[i].w, w.w, a);
        }
    }
}

// RAGGED: ranges that no piece divides, whose last piece stops at the range's end instead of multiplying zeros
// (K = 400 in ranges of 52: 8 to 10 % less; the second loop costs the other ranges 2 to 5 %).
template <bool GATED, bool RAGGED>
__global__ void __launch_bounds__(GT_THREADS)
gemm_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ W2,
                 float* __restrict__ C, int M, int N, int K, long long lda, long long ldc, GateAct act,
                 int m_tiles, int range) {
    constexpr int WIDE = GATED ? GT_N / 2 : GT_N;      // outputs a row
    extern __shared__ __align__(16) float gs_smem[];
    const int tid = threadIdx.x;
    const int rank = blockIdx.x & 7, tile = blockIdx.x >> 3;
    const int n0 = tile / m_tiles * WIDE, m0 = tile % m_tiles * GT_M;
    const int k_from = min(K, rank * range), k_to = min(K, k_from + range);
    const int pieces = (k_to - k_from + GT_K - 1) / GT_K;
    // rows GT_M .. of a stage are the weight's (the gated form's second weight's from GT_M + 64 on)
    auto fill = [&](int t, int from, int to) {         // rows from .. to - 1
        float* dst = gs_smem + (t % GT_STAGES) * GT_STAGE;
        const int k = k_from + t * GT_K + (tid & 3) * 4;
#pragma unroll
        for (int r = from + tid / 4; r < to; r += GT_THREADS / 4) {
            const bool of_x = r < GT_M;
            const int o = r - GT_M, half = GATED && o >= WIDE;
            const int at = of_x ? m0 + r : n0 + (half ? o - WIDE : o);
            const bool there = k < k_to && at < (of_x ? M : N);
            const float* src = of_x ? A : half ? W2 : W;
            gs_copy16(dst + r * GT_PITCH + (tid & 3) * 4,
                      src + (there ? (size_t)at * (of_x ? lda : (long long)K) + k : 0), there);
        }
    };
#pragma unroll
    for (int t = 0; t < GT_STAGES - 1; ++t)
        if (t < pieces) fill(t, GT_M, GT_M + GT_N);
    pdl_wait();
    pdl_launch_next();
#pragma unroll
    for (int t = 0; t < GT_STAGES - 1; ++t) {
        if (t < pieces) fill(t, 0, GT_M);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int tn = tid & 15, tm = tid >> 4;            // rows tm + 8 i of x, tn + 16 j of the weight
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    for (int t = 0; t < pieces; ++t) {
        asm volatile("cp.async.wait_group %0;" :: "n"(GT_STAGES - 2) : "memory");
        __syncthreads();                               // piece t is there, everybody is past t - 1
        if (t + GT_STAGES - 1 < pieces) fill(t + GT_STAGES - 1, 0, GT_M + GT_N);
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float* xs = gs_smem + (t % GT_STAGES) * GT_STAGE + tm * GT_PITCH;
        const float* ws = gs_smem + (t % GT_STAGES) * GT_STAGE + (GT_M + tn) * GT_PITCH;
        const int len = k_to - (k_from + t * GT_K);
        if (!RAGGED || len >= GT_K) {
#pragma unroll
            for (int k = 0; k < GT_K; k += 4) gt_four(acc, xs, ws, k);
        } else {
#pragma unroll 1
            for (int k = 0; k < len; k += 4) gt_four(acc, xs, ws, k);
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) gs_smem[(tm + 8 * i) * GT_N + tn + 16 * j] = acc[i][j];
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    // thread tid adds column tid of rows rank * 8 .. + 7 (the gated form: both weights' sums of a
    // column, four of the rows)
    const int col = tid % WIDE, n = n0 + col;
#pragma unroll 2
    for (int i = tid / WIDE; i < 8; i += GT_THREADS / WIDE) {
        const int m = rank * 8 + i;
        float v[2];
#pragma unroll
        for (int h = 0; h < (GATED ? 2 : 1); ++h) {
            float p[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) p[r] = gs_peer(gs_smem + m * GT_N + h * WIDE + col, r);
            v[h] = ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
        }
        if (n < N && m0 + m < M) C[(size_t)(m0 + m) * ldc + n] = finish<GATED>(v[0], v[GATED], act);
    }
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

struct GsArgs {
    const void *A, *W, *W2;
    void* C;
    int M, N, K;
    long long lda, ldc;
    GateAct act;
    cudaStream_t stream;
};

// BM == GT_M: tiles, else a warp's rows.
template <bool GATED, int BM, int R, bool DEEP = false>
static int launch_f32(const GsArgs& a) {
    constexpr bool TILE = BM == GT_M;
    constexpr int MATS = GATED ? 2 : 1, CL = TILE ? 8 : 4 / R;
    constexpr int WIDE = TILE ? GT_N / MATS : GS_ROWS;
    constexpr size_t smem = sizeof(float) * (TILE ? GT_STAGES * GT_STAGE
                                                  : GS_WARPS * gs_stages(MATS, BM, DEEP) * gs_stage_floats(MATS, BM));
    const long long m_tiles = (a.M + BM - 1) / BM, n_tiles = (a.N + WIDE - 1) / WIDE;
    AGV_REQUIRE(m_tiles * n_tiles * CL <= 0x7fffffffLL, "linear: M=%d N=%d exceed the grid limit", a.M, a.N);
    const int range = ((a.K + 7) / 8 + 3) / 4 * 4;
    void (*kern)(const float*, const float*, const float*, float*, int, int, int, long long, long long, GateAct,
                 int, int);
    if constexpr (TILE) kern = range % GT_K ? gemm_tile_kernel<GATED, true> : gemm_tile_kernel<GATED, false>;
    else kern = gemm_rows_kernel<GATED, BM, R, DEEP>;
    if (smem > 48 * 1024)
        AGV_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    agv_launch_cluster(kern, dim3((unsigned)(m_tiles * n_tiles * CL)), TILE ? GT_THREADS : GS_WARPS * 32, smem,
                       a.stream, dim3(CL), (const float*)a.A, (const float*)a.W, (const float*)a.W2, (float*)a.C,
                       a.M, a.N, a.K, a.lda, a.ldc, a.act, (int)m_tiles, range);
    AGV_LAUNCH_OK(TILE ? "gemm_tile_kernel" : "gemm_rows_kernel");
    return 0;
}

// R: a warp each where the groups of 32 weight rows are few or K is long (288 k a range keep a
// warp's ring busy), else two or four ranges a warp.  3 rows of x, us for R = 1, 2, 4:
// 1536 x 1152 12, 14, 19; 6912 x 1152 21, 18, 23; gated 35, 31, 27; 262144 x 1152 298, 258, 242;
// 10240 x 2560 35, 37, 39; 1152 x 6912 23, 40, 80.
// With up to four rows of x and 64 groups a warp keeps eight pieces under way instead of four: such a launch
// is at most 256 CTAs, all resident with 82 KB each, and four pieces are too few bytes for their trips to HBM
// (us, 1152 x 6912 19.1 -> 14.7, 1536 x 4096 12.0 -> 10.2, 2048 x 2304 8.0 -> 7.4, 256 x 10240 24.7 -> 18.5).
// More groups would need a second round (2304 x 2304 1.46 times the time with eight, 8192 x 4096 1.28), a gated pair
// takes 156 KB a CTA (1.6 to 2 times), eight rows gain nothing (0.96 to 1.08), and a walk of up to four pieces
// (K of 1,024) does from 57 groups on (1.02 to 1.05).
template <bool GATED, int BM>
static int launch_rows(const GsArgs& a) {
    const int pieces = (a.N + GS_ROWS - 1) / GS_ROWS * (GATED ? 2 : 1);
    if (pieces <= 128 || a.K >= 2304) {
        if constexpr (!GATED && BM == 4)
            if (pieces <= (a.K > 1024 ? 64 : 56)) return launch_f32<GATED, BM, 1, true>(a);
        return launch_f32<GATED, BM, 1>(a);
    }
    if constexpr (BM <= 16)
        if (pieces > 400) return launch_f32<GATED, BM, 4>(a);
    return launch_f32<GATED, BM, 2>(a);
}

template <typename TA, typename TW, typename TO, bool GATED>
static int launch_any(const GsArgs& a) {
    const dim3 grid((a.N + GA_N - 1) / GA_N, (a.M + GA_M - 1) / GA_M);
    agv_launch(gemm_any_kernel<TA, TW, TO, GATED>, grid, 256, 0, a.stream, (const TA*)a.A, (const TW*)a.W,
               (const TW*)a.W2, (TO*)a.C, a.M, a.N, a.K, a.lda, a.ldc, a.act);
    AGV_LAUNCH_OK("gemm_any_kernel");
    return 0;
}

// A K below this has ranges too short for a ring to fill (2048 x 256, 2,048 rows: 107 us either way;
// x 64: 34 us with one chain, 83 with eight).  At 384 many rows of a gated pair lose up to 9 % (4,096 outputs,
// 2,048 rows; at 400, whose ranges end inside a piece, a third) and few rows take a seventh (three rows 46 -> 7 us).  Which kernels a weight goes to follows
// from K and the alignment alone, so that a row's sums have one order whatever the number of rows.
constexpr int GS_MIN_K = 384;

template <bool GATED>
static int launch_gemm(const GsArgs& a, int in_dtype, int out_dtype) {
    if (in_dtype == AGV_F32 && out_dtype == AGV_F32) {
        const bool pieces = a.K % 4 == 0 && a.lda % 4 == 0 && agv_aligned(a.A, 16) && agv_aligned(a.W, 16) &&
                            agv_aligned(a.W2, 16);
        if (!pieces || a.K < GS_MIN_K) return launch_any<float, float, float, GATED>(a);
        if (a.M <= 4) return launch_rows<GATED, 4>(a);
        if (a.M <= 8) return launch_rows<GATED, 8>(a);
        if (a.M <= 16) return launch_rows<GATED, 16>(a);
        if (a.M <= 32) return launch_rows<GATED, 32>(a);
        return launch_f32<GATED, GT_M, 1>(a);
    }
    if (in_dtype == AGV_BF16 && out_dtype == AGV_BF16)
        return launch_any<__nv_bfloat16, __nv_bfloat16, __nv_bfloat16, GATED>(a);
    if (in_dtype == AGV_BF16 && out_dtype == AGV_F32)
        return launch_any<__nv_bfloat16, __nv_bfloat16, float, GATED>(a);
    return agv_fail(-1, "linear: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
}

// x: [M, K] with row stride lda; w (and w2 for the gated form): [N, K] dense;
// out: [M, N] with row stride ldc.  in_dtype is the dtype of x and of the
// weights; out_dtype may be 32-bit for a bfloat16 product (logits).
AGV_API int agv_linear_simt(const void* x, const void* w, const void* w2, void* out, int M, int N,
                            int K, long long lda, long long ldc, int in_dtype, int out_dtype,
                            int act_kind, float act_alpha, float act_limit, cudaStream_t stream) {
    const GateAct act{act_kind, act_alpha, act_limit};
    AGV_REQUIRE(M >= 0 && N > 0 && K > 0, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
    AGV_REQUIRE(lda >= K && ldc >= N, "linear: row strides %lld, %lld shorter than rows", lda, ldc);
    AGV_REQUIRE(w2 ? gate_act_ok(act) : act_kind >= 0 && act_kind <= AGV_ACT_GELU_ERF,
                "linear: activation %d does not go with this form of the product", act_kind);
    AGV_REQUIRE((long long)((M + GA_M - 1) / GA_M) <= 65535, "linear: M=%d exceeds the grid limit", M);
    if (M == 0) return 0;
    const GsArgs a{x, w, w2, out, M, N, K, lda, ldc, act, stream};
    return w2 ? launch_gemm<true>(a, in_dtype, out_dtype) : launch_gemm<false>(a, in_dtype, out_dtype);
}
