// The gated delta rule with a decay per key channel, as a recurrent mixer's kernels.
//
// A token's row of the stacked projection is  q | k | v | b | a1 | g1  (G*d, G*d, H*dv, H, ra
// and rg wide).  q, k and v pass a short causal convolution over time, channel by channel
// (``taps`` weights a channel, the last one the current token's; zeros before the start of a
// sequence), and silu.  Every q and k head becomes a unit vector (x / sqrt(sum x^2 + eps_unit)),
// q times a constant besides.  beta = sigmoid(b), one per head.  a1 and g1 are low-rank
// bottlenecks: a = W_a2 a1 and the gate W_g2 g1 are products of their own between the
// kernels here.  With the decay  g = exp(neg_a[h] * softplus(a + dt_bias))  per head and key
// channel, a head's state S [d, dv] goes
//
//      S <- diag(g) S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
//
// token by token (the read-out sees the token's own write), query/key head h / (H / G)
// serving head h.  The head's o is divided by its root mean square (eps_out), multiplied by a
// weight [dv] and by sigmoid(gate), and rounded to the compute dtype for the output product.
//
// The columns of S are independent recurrences over d-vectors, so the scan gives every column
// (or two) to a group of L lanes that hold 16 rows of it each in registers; the two dot products of a
// token are finished with L-wide shuffles.  A sequence's tokens run in order; sequences,
// heads and groups of columns run side by side.  The state of a sequence (S of every head,
// and the last taps - 1 inputs of the convolution) lives in 32-bit in the sequence's slot of
// the fixed-size state and is read at the start of a step and written at its end, so a
// prompt and a decoded token differ only in the form of the kernels that does their work fastest.
//
// 32-bit throughout: sums over partial products, the convolution, silu, unit norms, beta, the
// decay, the state and the recurrence, the output norm and the gate's sigmoid.
#include "common.cuh"
#include "row_in.cuh"

namespace {

constexpr int DL_R = 16;           // rows of a column a lane holds
constexpr int DL_MAX_TAPS = 16;

struct DeltaDims {
    int G, H, d, dv, taps, ra, rg;
    __host__ __device__ int nq() const { return G * d; }
    __host__ __device__ int nv() const { return H * dv; }
    __host__ __device__ int C() const { return 2 * G * d + H * dv; }      // convolved channels
    __host__ __device__ int W() const { return C() + H + ra + rg; }
};

// Where a step's sequences keep their state.
struct DeltaState {
    float* state;              // [n_slots, stride]
    long long stride;
    long long conv_off;        // the convolution's inputs [taps - 1, C] start here; S [H, dv, d] at 0
    const int* slots;          // [B]; negative: padding entry
    const int* cu;             // [B + 1] first token of each entry
    const int* seq_index;      // [T]
    const int* positions;      // [T]
};

__device__ __forceinline__ float silu_f(float t) { return t / (1.0f + expf(-t)); }
__device__ __forceinline__ float sigmoid_f(float t) { return 1.0f / (1.0f + expf(-t)); }
__device__ __forceinline__ float softplus_f(float t) {
    return t > 20.0f ? t : log1pf(expf(t));
}

// ------------------------------------------------------------------ prepare
// Two forms, a CTA a token (any sizes) and a warp a head's or a piece of a row's channels (below).
// The convolution's inputs of a sequence are a ring by position: the input of position pp is
// row pp % (taps - 1) of the slot's [taps - 1, C] block, so a step writes the rows of its own
// last taps - 1 positions and moves nothing.
//
// One CTA per token.  The token's row of the stacked product comes into shared memory first
// (all its loads in flight at once), earlier tokens of the same step are read in place.
// fused_state: the CTA's token is the only one its sequence brings (a decode step), so it
// also stores its inputs in the ring.
template <typename T>
__global__ void __launch_bounds__(256)
delta_prepare_kernel(RowIn<T> in, DeltaDims dm, DeltaState st, const float* __restrict__ conv_w,
                     float eps_unit, float q_mult, int fused_state, float* __restrict__ qkv,
                     float* __restrict__ beta, T* __restrict__ low_a, T* __restrict__ low_g) {
    pdl_wait();
    pdl_launch_next();
    extern __shared__ float buf[];               // [C] convolved and activated channels
    const int t = blockIdx.x;
    const int b = st.seq_index[t];
    const int slot = st.slots[b];
    if (slot < 0) return;
    const int C = dm.C(), nq = dm.nq(), taps = dm.taps, R = taps - 1;
    float* rowbuf = buf + C;                     // [W] the token's row, 32-bit
    const int p = st.positions[t];
    const int first = st.cu[b];                  // first token of the sequence in this step
    const int p0 = p - (t - first);              // its position
    in.load(t, rowbuf);
    {
        const float* __restrict__ cs = st.state + (size_t)slot * st.stride + st.conv_off;
#pragma unroll 4
        for (int c = threadIdx.x; c < C; c += blockDim.x) {
            const float* w = conv_w + (size_t)c * taps;
            float acc = 0.f;
            // oldest input first; input p - k meets weight taps - 1 - k
            for (int k = R; k >= 1; --k) {
                const int pp = p - k;
                float x = 0.f;
                if (pp >= p0) x = in.at(t - k, c);
                else if (pp >= 0) x = cs[(size_t)(pp % R) * C + c];
                acc = fmaf(w[R - k], x, acc);
            }
            buf[c] = silu_f(fmaf(w[R], rowbuf[c], acc));
        }
    }
    if (fused_state && R > 0) {
        // (the row of position p is the one position p - R had: read above by this thread)
        float* cs = st.state + (size_t)slot * st.stride + st.conv_off + (size_t)(p % R) * C;
        for (int c = threadIdx.x; c < C; c += blockDim.x) cs[c] = rowbuf[c];
    }
    __syncthreads();
    // unit vectors: q heads, then k heads (2 G groups of d), a warp a group
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    float* orow = qkv + (size_t)t * C;
    for (int grp = warp; grp < 2 * dm.G; grp += nwarps) {
        const float* x = buf + (size_t)grp * dm.d;
        float ss = 0.f;
        for (int i = lane; i < dm.d; i += 32) ss = fmaf(x[i], x[i], ss);
        ss = warp_sum(ss);
        const float r = (1.0f / sqrtf(ss + eps_unit)) * (grp < dm.G ? q_mult : 1.0f);
        for (int i = lane; i < dm.d; i += 32) orow[(size_t)grp * dm.d + i] = x[i] * r;
    }
    for (int c = 2 * nq + threadIdx.x; c < C; c += blockDim.x) orow[c] = buf[c];
    for (int h = threadIdx.x; h < dm.H; h += blockDim.x)
        beta[(size_t)t * dm.H + h] = sigmoid_f(rowbuf[C + h]);
    for (int i = threadIdx.x; i < dm.ra; i += blockDim.x)
        low_a[(size_t)t * dm.ra + i] = from_f32<T>(rowbuf[C + dm.H + i]);
    for (int i = threadIdx.x; i < dm.rg; i += blockDim.x)
        low_g[(size_t)t * dm.rg + i] = from_f32<T>(rowbuf[C + dm.H + dm.ra + i]);
}

// The same where the row comes in 32-bit in whole 16-byte pieces, with two to four taps and heads of
// up to 256: a warp has R tokens of one q or k head, of 128 NJ columns of v, or of 32 of the last
// columns (b, a1, g1), a lane four neighbouring channels, whose inputs slide through registers.
// Weights and the step's arrays are asked for before the dependency wait, the ring after it: the kernel
// before may be the one that writes it (another step's, a call apart).
//
// A decode step is bound by trips to memory one after the other: a CTA a token walked its 3,216
// columns in a dozen of them, 35 us for 8 tokens (G 4, H 16, heads of 128, eight partial sums);
// 29 warps a token make two, 4.7 us.  A prompt is bound by its rows (126 MB for 5,120 tokens, 20
// us): 191 us -> 108 with R = 8, which reads a row once instead of once a tap.
template <typename T, int TAPS, int NJ, int R>
__global__ void __launch_bounds__(128)
delta_prepare_rows_kernel(RowIn<float> in, DeltaDims dm, DeltaState st, int n_tokens, int n_seg,
                          const float* __restrict__ conv_w, float eps_unit, float q_mult, int fused_state,
                          float* __restrict__ qkv, float* __restrict__ beta, T* __restrict__ low_a,
                          T* __restrict__ low_g) {
    constexpr int RING = TAPS - 1, SW = NJ * 128;
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    const int tile = (int)(w / n_seg), seg = (int)(w - (long long)tile * n_seg);
    const int t0 = tile * R;
    const int C = dm.C(), nq = dm.nq(), nv = dm.nv();
    const int v_seg = (nv + SW - 1) / SW, conv_seg = 2 * dm.G + v_seg;
    if (t0 >= n_tokens) return;
    if (seg >= conv_seg) {
        pdl_wait();
        pdl_launch_next();
        const int e = (seg - conv_seg) * 32 + lane;
        if (e >= dm.H + dm.ra + dm.rg) return;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            const int t = t0 + i;
            if (t >= n_tokens) break;
            if (st.slots[st.seq_index[t]] < 0) continue;
            const float x = in.at(t, C + e);
            if (e < dm.H) beta[(size_t)t * dm.H + e] = sigmoid_f(x);
            else if (e < dm.H + dm.ra) low_a[(size_t)t * dm.ra + e - dm.H] = from_f32<T>(x);
            else low_g[(size_t)t * dm.rg + e - dm.H - dm.ra] = from_f32<T>(x);
        }
        return;
    }
    const bool head = seg < 2 * dm.G;
    const int c0 = head ? seg * dm.d : 2 * nq + (seg - 2 * dm.G) * SW;
    const int width = head ? dm.d : min(SW, nv - (seg - 2 * dm.G) * SW);
    float wv[NJ][4 * TAPS];
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        const int ch = j * 128 + lane * 4;
#pragma unroll
        for (int k = 0; k < TAPS; ++k) {
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ch < width) v = *reinterpret_cast<const float4*>(conv_w + (size_t)(c0 + ch) * TAPS + 4 * k);
            wv[j][4 * k] = v.x; wv[j][4 * k + 1] = v.y; wv[j][4 * k + 2] = v.z; wv[j][4 * k + 3] = v.w;
        }
    }
    int pos[R], slot[R], before[R];
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int t = min(t0 + i, n_tokens - 1), b = st.seq_index[t];
        pos[i] = st.positions[t];
        slot[i] = st.slots[b];
        before[i] = t - st.cu[b];
    }
    pdl_wait();
    pdl_launch_next();
    // the ring's rows before the tile's first token (later tokens of the tile that reach further
    // back than their sequence's first token in the step read it themselves, below)
    float4 old[NJ][RING];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int k = 1; k <= RING; ++k) {
            const int ch = j * 128 + lane * 4;
            old[j][k - 1] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (ch < width && slot[0] >= 0 && k > before[0] && pos[0] - k >= 0)
                old[j][k - 1] = *reinterpret_cast<const float4*>(
                    st.state + (size_t)slot[0] * st.stride + st.conv_off + (size_t)((pos[0] - k) % RING) * C + c0 + ch);
        }
    float4 xs[NJ][R + RING];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int i = 0; i < R + RING; ++i) {
            const int t = t0 - RING + i, ch = j * 128 + lane * 4;
            float4 a = make_float4(0.f, 0.f, 0.f, 0.f);
            // (one token a tile: earlier tokens of the step are other sequences')
            if ((R > 1 || i == RING) && t >= 0 && t < n_tokens && ch < width) {
                if (in.part) {
                    const float* p = in.part + (size_t)t * in.W + c0 + ch;
#pragma unroll 8
                    for (int sp = 0; sp < in.n_splits; ++sp) {
                        const float4 v = *reinterpret_cast<const float4*>(p + (size_t)sp * in.split_stride);
                        a.x += v.x; a.y += v.y; a.z += v.z; a.w += v.w;
                    }
                } else {
                    a = *reinterpret_cast<const float4*>(in.row + (size_t)t * in.ld + c0 + ch);
                }
            }
            xs[j][i] = a;
        }
    // a tile whose every token finds its whole past in the step: products and sums alone
    bool plain = R > 1 && t0 + R <= n_tokens && !fused_state;
#pragma unroll
    for (int i = 0; i < R; ++i) plain = plain && slot[i] >= 0 && before[i] >= RING;
    if (R > 1 && plain) {
        const float mult = seg < dm.G ? q_mult : 1.0f;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            float y[NJ][4], ss = 0.f;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int k = RING; k >= 0; --k) {          // oldest input first
                    const float4 x = xs[j][RING + i - k];
                    acc[0] = fmaf(wv[j][RING - k], x.x, acc[0]);
                    acc[1] = fmaf(wv[j][TAPS + RING - k], x.y, acc[1]);
                    acc[2] = fmaf(wv[j][2 * TAPS + RING - k], x.z, acc[2]);
                    acc[3] = fmaf(wv[j][3 * TAPS + RING - k], x.w, acc[3]);
                }
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    y[j][e] = silu_f(acc[e]);
                    ss = fmaf(y[j][e], y[j][e], ss);
                }
            }
            const float r = head ? (1.0f / sqrtf(warp_sum(ss) + eps_unit)) * mult : 1.f;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const int ch = j * 128 + lane * 4;
                if (ch < width)
                    *reinterpret_cast<float4*>(qkv + (size_t)(t0 + i) * C + c0 + ch) =
                        make_float4(y[j][0] * r, y[j][1] * r, y[j][2] * r, y[j][3] * r);
            }
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < R; ++i) {
        const int t = t0 + i;
        if (t >= n_tokens) break;
        if (slot[i] < 0) continue;
        const float* ring = st.state + (size_t)slot[i] * st.stride + st.conv_off + c0;
        float y[NJ][4], ss = 0.f;
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int ch = j * 128 + lane * 4;
            float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = RING; k >= 1; --k) {              // oldest input first
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (R > 1 && k <= before[i]) x = xs[j][RING + i - k];
                else if (i == 0) x = old[j][k - 1];
                else if (pos[i] - k >= 0 && ch < width)
                    x = *reinterpret_cast<const float4*>(ring + (size_t)((pos[i] - k) % RING) * C + ch);
                const float xe[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[e] = fmaf(wv[j][e * TAPS + RING - k], xe[e], acc[e]);
            }
            const float4 x = xs[j][RING + i];
            const float xe[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                y[j][e] = silu_f(fmaf(wv[j][e * TAPS + RING], xe[e], acc[e]));
                ss = fmaf(y[j][e], y[j][e], ss);
            }
            if (fused_state && ch < width)                 // (the row that position p - RING had)
                *reinterpret_cast<float4*>(st.state + (size_t)slot[i] * st.stride + st.conv_off +
                                           (size_t)(pos[i] % RING) * C + c0 + ch) = x;
        }
        float r = 1.f;
        if (head) r = (1.0f / sqrtf(warp_sum(ss) + eps_unit)) * (seg < dm.G ? q_mult : 1.0f);
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            const int ch = j * 128 + lane * 4;
            if (ch < width)
                *reinterpret_cast<float4*>(qkv + (size_t)t * C + c0 + ch) =
                    make_float4(y[j][0] * r, y[j][1] * r, y[j][2] * r, y[j][3] * r);
        }
    }
}

// The convolution's inputs after a step of several tokens a sequence: the step's last
// taps - 1 positions go to their rows of the ring (fewer, if the step is shorter: the rows of
// earlier positions stay).  One CTA per sequence, a thread a channel; it runs after the
// prepare kernel, which reads the inputs of before the step.
template <typename T>
__global__ void __launch_bounds__(256)
delta_conv_state_kernel(RowIn<T> in, DeltaDims dm, DeltaState st) {
    pdl_wait();
    pdl_launch_next();
    const int b = blockIdx.x;
    const int slot = st.slots[b];
    if (slot < 0) return;
    const int C = dm.C(), R = dm.taps - 1;
    const int first = st.cu[b], n = st.cu[b + 1] - first;
    if (n <= 0 || R <= 0) return;
    const int p0 = st.positions[first], len = p0 + n;
    const int from = len - R > p0 ? len - R : p0;
    float* cs = st.state + (size_t)slot * st.stride + st.conv_off;
    for (int c = threadIdx.x; c < C; c += blockDim.x)
        for (int pp = from; pp < len; ++pp)
            cs[(size_t)(pp % R) * C + c] = in.at(first + pp - p0, c);
}

// --------------------------------------------------------------------- scan
// grid (column groups, H, B); a CTA has CC columns of one head of one sequence, L lanes a
// column (L a power of two, L * 16 >= d), thread = column * L + lane.  The tokens of the
// sequence come through shared memory TCH at a time: k, q and the decay of the head's key
// channels (padded with zeros to L * 16 rows, which keeps the padded rows of S at zero), the
// CTA's columns of v, and beta.  L is a template parameter: the shuffle rounds are unrolled.
// A lane's 16 rows are four quads, quad i of lane l being rows (i * L + l) * 4 .. + 3: the
// lanes of a column then read consecutive 16 bytes of a token's row, free of bank conflicts
// (the columns of a warp read the same addresses).
struct ScanArgs {
    const float* qkv;          // [T, C]: q | k | v, prepared
    const float* beta;         // [T, H]
    const float* a;            // [T, H * d]: the decay's pre-activation, without its bias
    const float* dt_bias;      // [H * d]
    const float* neg_a;        // [H]: -exp(A_log)
    float* out;                // [T, H * dv]
    int L, CC, TCH;
    // what does not depend on the state, made by the launch before, [T, H, L * 16] each with
    // zeros in the padding, and k . q [T, H]
    float *wk, *wg, *wgk, *wgq, *wkq;
};

// What a token's step needs besides the state, for every head: k, the decay g = exp(neg_a *
// softplus(a + bias)), g * k, g * q and k . q.  A warp a (token, head); rows of Dp = L * 16
// floats, the padding zero, so that the scan copies them 16 bytes at a time.
__global__ void __launch_bounds__(256)
delta_decay_kernel(ScanArgs a, DeltaDims dm, int T, int Dp) {
    pdl_wait();
    pdl_launch_next();
    const int lane = threadIdx.x & 31;
    const long long w = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (w >= (long long)T * dm.H) return;
    const int t = (int)(w / dm.H), h = (int)(w - (long long)t * dm.H), g = h / (dm.H / dm.G);
    const int d = dm.d;
    const float* q = a.qkv + (size_t)t * dm.C() + (size_t)g * d;
    const float* k = q + dm.nq();
    const float* pre = a.a + ((size_t)t * dm.H + h) * d;
    const float* bias = a.dt_bias + (size_t)h * d;
    const float na = a.neg_a[h];
    const size_t o = (size_t)w * Dp;
    float s = 0.f;
    for (int r = lane; r < Dp; r += 32) {
        float kv = 0.f, gv = 0.f, qv = 0.f;
        if (r < d) {
            kv = k[r];
            qv = q[r];
            gv = expf(na * softplus_f(pre[r] + bias[r]));
        }
        a.wk[o + r] = kv;
        a.wg[o + r] = gv;
        a.wgk[o + r] = gv * kv;
        a.wgq[o + r] = gv * qv;
        s = fmaf(kv, qv, s);
    }
    s = warp_sum(s);
    if (lane == 0) a.wkq[w] = s;
}

// A 4-byte asynchronous copy into shared memory (the sources are rows of 32-bit tensors at
// offsets that need not be multiples of 16 bytes).
__device__ __forceinline__ void cp_async_f32(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;"
                 :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                 :: "r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// The tokens come through two buffers: while the lanes run the recurrence over one, the next
// TCH tokens' k, q, decay pre-activation, v and beta are on their way (asynchronous copies),
// so the trip to L2 or HBM is paid once a sequence, not once a buffer.  What does not depend
// on the state was made by the launch before for all tokens at once: the decay g, g * k,
// g * q and the token's k . q.  With them a token is one round of dot products,
//
//      a = (g S)^T k = sum_r S_r (g k)_r      r = (g S)^T q = sum_r S_r (g q)_r
//      u = beta (v - a);    o = r + (k . q) u;    S <- g S + k u
//
// the same sums as  S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q  with the
// read-out split into the part the state had and the token's own write: one round of
// shuffles a token instead of two, and the state's update off the output's path.
struct ScanBuf {
    float *k, *gk, *gq, *g, *v, *beta, *kq;
    __device__ ScanBuf(float* base, int TCH, int Dp, int CC) {
        k = base;
        gk = k + (size_t)TCH * Dp;       // (q arrives in gq's place, the pre-activation in g's)
        gq = gk + (size_t)TCH * Dp;
        g = gq + (size_t)TCH * Dp;
        v = g + (size_t)TCH * Dp;
        beta = v + (size_t)TCH * CC;
        kq = beta + TCH;
    }
};
__host__ __device__ inline size_t scan_buf_floats(int TCH, int Dp, int CC) {
    return ((size_t)TCH * (4 * Dp + CC + 2) + 3) / 4 * 4;      // (16-byte rows in the next buffer)
}

// A lane's rows of CPT columns (CC apart): a piece of a token's row read once serves them all.  One column's
// rows are single values; two columns' are pairs, two rows to a register pair.  What bounds it are a token's
// reads of k, g, g k and g q (16 of 16 bytes a lane), the sums over the lanes and the wait for u, token after
// token, behind the longest sequence; a step of one token a sequence (STEP) is bound by the trip to memory.
//
// 8 sequences of 256 to 1,024 tokens, 16 heads of 128 x 128: 905 us with one column a lane and the sequences
// as they come; 644 with two columns and the longest first (four: 620, but a step of 287 tokens lost what that
// gained).  One column in pairs is slower, a chain of half as many but slower operations: one sequence of
// 1,024 tokens, 8 heads of 64 x 64 310 us against 224.  Registers: a prompt's loads of a token are asked for
// together where there are enough (the compiler, left alone, kept to 72 and 80: 705 us for the eight sequences
// above, 670 with 128); a STEP has no second token and wants warps instead (64 sequences, 32 heads of 128 x
// 128: 92 us with 100 registers, 76 with 64).
constexpr int scan_ctas(int cpt, bool step) { return step ? 7 : cpt == 1 ? 1 : 4; }
template <int L, int CPT, bool STEP>
__global__ void __launch_bounds__(128, scan_ctas(CPT, STEP))
delta_scan_kernel(ScanArgs a, DeltaDims dm, DeltaState st) {
    pdl_wait();
    extern __shared__ float smem[];
    // the longest sequences of a prompt step begin first: this CTA's is the blockIdx.z-th longest
    int b = blockIdx.z;
    if (!STEP && gridDim.z <= blockDim.x) {
        __shared__ int ranked;
        const int e = threadIdx.x, B = gridDim.z;
        if (e < B) {
            const int mine = st.cu[e + 1] - st.cu[e];
            int rank = 0;
            for (int j = 0; j < B; ++j) {
                const int other = st.cu[j + 1] - st.cu[j];
                rank += other > mine || (other == mine && j < e);
            }
            if (rank == (int)blockIdx.z) ranked = e;
        }
        __syncthreads();
        b = ranked;
    }
    const int slot = st.slots[b];
    if (slot < 0) return;
    const int t0 = st.cu[b], n = st.cu[b + 1] - t0;
    if (n <= 0) return;
    const int h = blockIdx.y;
    const int d = dm.d, dv = dm.dv, C = dm.C(), nq = dm.nq();
    constexpr int Dp = L * DL_R, P = DL_R / 2, TOKENS = STEP ? 1 : 2;
    const int CC = a.CC, CW = CC * CPT, TCH = a.TCH;
    const int l = threadIdx.x & (L - 1);
    const int jc = threadIdx.x / L;
    const int j0 = blockIdx.x * CW + jc;               // and j0 + CC, ...
    bool live[CPT];
#pragma unroll
    for (int x = 0; x < CPT; ++x) live[x] = jc < CC && j0 + x * CC < dv;
    const size_t per = scan_buf_floats(TCH, Dp, CW);
    // (columns of v past dv are never copied: zero them once)
    for (size_t i = threadIdx.x; i < 2 * per; i += blockDim.x) smem[i] = 0.f;
    __syncthreads();

    auto fetch = [&](int c0, float* base) {
        const int m = min(TCH, n - c0);
        const ScanBuf sb(base, TCH, Dp, CW);
        // rows of Dp floats a token: tokens of a head lie H * Dp apart
        constexpr int Q = Dp / 4;
        for (int idx = threadIdx.x; idx < m * Q; idx += blockDim.x) {
            const int tt = idx / Q, c4 = (idx - tt * Q) * 4;
            const size_t src = ((size_t)(t0 + c0 + tt) * dm.H + h) * Dp + c4;
            const int dst = tt * Dp + c4;
            cp_async_16(sb.k + dst, a.wk + src);
            cp_async_16(sb.g + dst, a.wg + src);
            cp_async_16(sb.gk + dst, a.wgk + src);
            cp_async_16(sb.gq + dst, a.wgq + src);
        }
        for (int idx = threadIdx.x; idx < m * CW; idx += blockDim.x) {
            const int tt = idx / CW, c = idx - tt * CW;
            const int col = blockIdx.x * CW + c;
            if (col < dv)
                cp_async_f32(sb.v + idx, a.qkv + (size_t)(t0 + c0 + tt) * C + 2 * nq + (size_t)h * dv + col);
        }
        for (int tt = threadIdx.x; tt < m; tt += blockDim.x) {
            cp_async_f32(sb.beta + tt, a.beta + (size_t)(t0 + c0 + tt) * dm.H + h);
            cp_async_f32(sb.kq + tt, a.wkq + (size_t)(t0 + c0 + tt) * dm.H + h);
        }
        cp_async_commit();
    };

    // S: single values where a lane has one column, else pairs
    float S1[CPT == 1 ? DL_R : 1];
    f32x2 S[CPT == 1 ? 1 : CPT][P];
    float* srow[CPT];
    fetch(0, smem);
#pragma unroll
    for (int x = 0; x < CPT; ++x) {
        srow[x] = st.state + (size_t)slot * st.stride + ((size_t)h * dv + (live[x] ? j0 + x * CC : 0)) * d;
#pragma unroll
        for (int i = 0; i < P; ++i) {
            const int r = ((i >> 1) * L + l) * 4 + (i & 1) * 2;
            const float lo = live[x] && r < d ? srow[x][r] : 0.f, hi = live[x] && r + 1 < d ? srow[x][r + 1] : 0.f;
            if constexpr (CPT == 1) { S1[2 * i] = lo; S1[2 * i + 1] = hi; }
            else S[x][i] = pack2(lo, hi);
        }
    }
    int cur = 0;
    for (int c0 = 0; c0 < n; c0 += TCH, cur ^= 1) {
        const int m = min(TCH, n - c0);
        const ScanBuf sb(smem + (size_t)cur * per, TCH, Dp, CW);
        // (the other buffer was read in the round before, which ended with a barrier)
        if (c0 + TCH < n) {
            fetch(c0 + TCH, smem + (size_t)(cur ^ 1) * per);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
        const float* pk = sb.k + l * 4;
        const float* pgk = sb.gk + l * 4;
        const float* pgq = sb.gq + l * 4;
        const float* pg = sb.g + l * 4;
        const float* pv = sb.v + (jc < CC ? jc : 0);
        float* po = a.out + (size_t)(t0 + c0) * dm.H * dv + (size_t)h * dv + j0;
#pragma unroll TOKENS
        for (int tt = 0; tt < m; ++tt) {
            if constexpr (CPT == 1) {
                float gk[DL_R], gq[DL_R], kk[DL_R], gg[DL_R];
#pragma unroll
                for (int i = 0; i < DL_R / 4; ++i) {
                    const float4 x = reinterpret_cast<const float4*>(pgk)[i * L];
                    const float4 y = reinterpret_cast<const float4*>(pgq)[i * L];
                    gk[4 * i] = x.x; gk[4 * i + 1] = x.y; gk[4 * i + 2] = x.z; gk[4 * i + 3] = x.w;
                    gq[4 * i] = y.x; gq[4 * i + 1] = y.y; gq[4 * i + 2] = y.z; gq[4 * i + 3] = y.w;
                }
                float ac[4] = {0.f, 0.f, 0.f, 0.f}, rc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int i = 0; i < DL_R; ++i) {
                    ac[i & 3] = fmaf(S1[i], gk[i], ac[i & 3]);
                    rc[i & 3] = fmaf(S1[i], gq[i], rc[i & 3]);
                }
#pragma unroll
                for (int i = 0; i < DL_R / 4; ++i) {
                    const float4 x = reinterpret_cast<const float4*>(pk)[i * L];
                    const float4 y = reinterpret_cast<const float4*>(pg)[i * L];
                    kk[4 * i] = x.x; kk[4 * i + 1] = x.y; kk[4 * i + 2] = x.z; kk[4 * i + 3] = x.w;
                    gg[4 * i] = y.x; gg[4 * i + 1] = y.y; gg[4 * i + 2] = y.z; gg[4 * i + 3] = y.w;
                }
                float acc = (ac[0] + ac[1]) + (ac[2] + ac[3]);
                float rr = (rc[0] + rc[1]) + (rc[2] + rc[3]);
#pragma unroll
                for (int o = 1; o < L; o <<= 1) {
                    acc += __shfl_xor_sync(0xffffffffu, acc, o);
                    rr += __shfl_xor_sync(0xffffffffu, rr, o);
                }
#pragma unroll
                for (int i = 0; i < DL_R; ++i) gg[i] *= S1[i];         // g S: needs no u
                const float u = sb.beta[tt] * (*pv - acc);
                if (live[0] && l == 0) *po = fmaf(sb.kq[tt], u, rr);
#pragma unroll
                for (int i = 0; i < DL_R; ++i) S1[i] = fmaf(kk[i], u, gg[i]);
            } else {
                f32x2 ac[CPT][2], rc[CPT][2];
#pragma unroll
                for (int x = 0; x < CPT; ++x) ac[x][0] = ac[x][1] = rc[x][0] = rc[x][1] = 0;
#pragma unroll
                for (int i = 0; i < DL_R / 4; ++i) {
                    const ulonglong2 gk = reinterpret_cast<const ulonglong2*>(pgk)[i * L];
                    const ulonglong2 gq = reinterpret_cast<const ulonglong2*>(pgq)[i * L];
#pragma unroll
                    for (int x = 0; x < CPT; ++x) {
                        ac[x][0] = fma2(S[x][2 * i], gk.x, ac[x][0]);
                        ac[x][1] = fma2(S[x][2 * i + 1], gk.y, ac[x][1]);
                        rc[x][0] = fma2(S[x][2 * i], gq.x, rc[x][0]);
                        rc[x][1] = fma2(S[x][2 * i + 1], gq.y, rc[x][1]);
                    }
                }
                float acc[CPT], rr[CPT];
#pragma unroll
                for (int x = 0; x < CPT; ++x) {
                    float a0, a1, a2, a3, r0, r1, r2, r3;
                    unpack2(ac[x][0], a0, a1); unpack2(ac[x][1], a2, a3);
                    unpack2(rc[x][0], r0, r1); unpack2(rc[x][1], r2, r3);
                    acc[x] = (a0 + a1) + (a2 + a3);
                    rr[x] = (r0 + r1) + (r2 + r3);
                }
#pragma unroll
                for (int o = 1; o < L; o <<= 1)
#pragma unroll
                    for (int x = 0; x < CPT; ++x) {
                        acc[x] += __shfl_xor_sync(0xffffffffu, acc[x], o);
                        rr[x] += __shfl_xor_sync(0xffffffffu, rr[x], o);
                    }
                const float beta = sb.beta[tt], kq = sb.kq[tt];
                f32x2 uu[CPT];
#pragma unroll
                for (int x = 0; x < CPT; ++x) {
                    const float u = beta * (pv[x * CC] - acc[x]);
                    if (live[x] && l == 0) po[x * CC] = fmaf(kq, u, rr[x]);
                    uu[x] = pack2(u, u);
                }
#pragma unroll
                for (int i = 0; i < DL_R / 4; ++i) {
                    const ulonglong2 kk = reinterpret_cast<const ulonglong2*>(pk)[i * L];
                    const ulonglong2 gg = reinterpret_cast<const ulonglong2*>(pg)[i * L];
#pragma unroll
                    for (int x = 0; x < CPT; ++x) {
                        S[x][2 * i] = fma2(kk.x, uu[x], mul2(gg.x, S[x][2 * i]));
                        S[x][2 * i + 1] = fma2(kk.y, uu[x], mul2(gg.y, S[x][2 * i + 1]));
                    }
                }
            }
            pk += Dp; pgk += Dp; pgq += Dp; pg += Dp; pv += CW;
            po += (size_t)dm.H * dv;
        }
        __syncthreads();
    }
    pdl_launch_next();
#pragma unroll
    for (int x = 0; x < CPT; ++x)
        if (live[x])
#pragma unroll
            for (int i = 0; i < P; ++i) {
                const int r = ((i >> 1) * L + l) * 4 + (i & 1) * 2;
                float lo, hi;
                if constexpr (CPT == 1) { lo = S1[2 * i]; hi = S1[2 * i + 1]; }
                else unpack2(S[x][i], lo, hi);
                if (r < d) srow[x][r] = lo;
                if (r + 1 < d) srow[x][r + 1] = hi;
            }
}

// ---------------------------------------------------------------- read-out
// y[t, h, :] = o[t, h, :] / rms(o[t, h, :]) * w * sigmoid(gate[t, h, :]): L lanes a head (a warp, or
// eight for heads of up to 32 values), a lane V neighbouring columns at a time, whose o and gate are asked
// for together; it keeps NJ V of them and reads the rest again.  Bound by the trip to memory when decoding
// (8 tokens, 16 heads of 128: one warp of four a CTA went through four heads, two trips each, 7.4 us -> 2.4
// us), by the instructions in a prompt (5,120 tokens, 105 MB, 16 us of HBM: 46 -> 27).  There every head costs
// its warp's address, and columns that are not there their predicates: with the token by a 64-bit division and
// NJ = 4 it took 42; heads of 16 on a warp each 31, now 7.6.
template <typename T, int V, int NJ, int L>
__global__ void __launch_bounds__(128)
delta_out_kernel(const float* __restrict__ o, const float* __restrict__ gate,
                 const float* __restrict__ w, float eps, int n_tokens, int H, int dv,
                 const int* __restrict__ seq_index, const int* __restrict__ slots,
                 T* __restrict__ y) {
    constexpr int HEADS = 128 / L;                       // of a CTA
    const int lane = threadIdx.x % L;
    const unsigned h_ctas = (unsigned)(H + HEADS - 1) / HEADS, t = blockIdx.x / h_ctas;
    const int at = (int)(blockIdx.x - t * h_ctas) * HEADS + threadIdx.x / L;
    const int h = min(at, H - 1);                        // (lanes behind the last head store nothing)
    const bool pad = slots[seq_index[t]] < 0;            // a padding entry's row is zeros
    const size_t base = ((size_t)t * H + h) * dv;
    pdl_wait();
    pdl_launch_next();
    float ov[NJ * V], gv[NJ * V], ss = 0.f;
    auto load = [&](const float* p, float* to) {
        if constexpr (V == 4) {
            const float4 x = *reinterpret_cast<const float4*>(p);
            to[0] = x.x; to[1] = x.y; to[2] = x.z; to[3] = x.w;
        } else {
            to[0] = *p;
        }
    };
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        const int i = (j * L + lane) * V;
        if (i < dv) {
            load(o + base + i, ov + j * V);
            load(gate + base + i, gv + j * V);
#pragma unroll
            for (int e = 0; e < V; ++e) ss = fmaf(ov[j * V + e], ov[j * V + e], ss);
        }
    }
    for (int i = (NJ * L + lane) * V; i < dv; i += L * V)
#pragma unroll
        for (int e = 0; e < V; ++e) ss = fmaf(o[base + i + e], o[base + i + e], ss);
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    if (at >= H) return;
    const float r = 1.0f / sqrtf(ss / (float)dv + eps);
    auto store = [&](int i, const float* a, const float* g) {
        float v[V];
#pragma unroll
        for (int e = 0; e < V; ++e) v[e] = pad ? 0.f : a[e] * r * w[i + e] * sigmoid_f(g[e]);
        if constexpr (V == 4 && sizeof(T) == 2) {
            const __nv_bfloat162 lo = __floats2bfloat162_rn(v[0], v[1]), hi = __floats2bfloat162_rn(v[2], v[3]);
            uint2 b;
            b.x = *reinterpret_cast<const uint32_t*>(&lo);
            b.y = *reinterpret_cast<const uint32_t*>(&hi);
            *reinterpret_cast<uint2*>(y + base + i) = b;
        } else {
#pragma unroll
            for (int e = 0; e < V; ++e) y[base + i + e] = from_f32<T>(v[e]);
        }
    };
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
        const int i = (j * L + lane) * V;
        if (i < dv) store(i, ov + j * V, gv + j * V);
    }
    for (int i = (NJ * L + lane) * V; i < dv; i += L * V) store(i, o + base + i, gate + base + i);
}

}  // namespace

static int check_dims(const DeltaDims& dm) {
    AGV_REQUIRE(dm.G > 0 && dm.H > 0 && dm.d > 0 && dm.dv > 0 && dm.ra >= 0 && dm.rg >= 0,
                "delta: bad sizes");
    AGV_REQUIRE(dm.H % dm.G == 0, "delta: %d heads are not a multiple of %d query/key heads",
                dm.H, dm.G);
    AGV_REQUIRE(dm.taps >= 1 && dm.taps <= DL_MAX_TAPS, "delta: %d taps, at most %d", dm.taps,
                DL_MAX_TAPS);
    AGV_REQUIRE(dm.d <= 32 * DL_R, "delta: key heads of %d exceed %d", dm.d, 32 * DL_R);
    return 0;
}

// row: [T, W] with row stride ld (dtype), or part: [n_splits, T, W] 32-bit partial sums, W =
// 2 G d + H dv + H + ra + rg.  conv_w: [2 G d + H dv, taps] 32-bit.  state: [n_slots,
// state_stride] 32-bit, the convolution's inputs [taps - 1, 2 G d + H dv] at conv_off (a ring:
// position pp in row pp % (taps - 1)).
// form: 0 the faster one, 1 the rows form, 2 a CTA a token.
// several != 0: sequences may bring more than one token (a prompt step); the convolution's
// inputs are then renewed by a launch of its own.  Outputs: qkv [T, 2 G d + H dv] and beta
// [T, H] 32-bit, low_a [T, ra] and low_g [T, rg] in dtype.
AGV_API int agv_delta_prepare(const void* row, long long ld, const float* part, int n_splits,
                              int dtype, int T, int B, int G, int H, int d, int dv, int taps,
                              int ra, int rg, const float* conv_w, float eps_unit, float q_mult,
                              float* state, long long state_stride, long long conv_off,
                              const int* slots, const int* cu, const int* seq_index,
                              const int* positions, int several, int form, float* qkv, float* beta,
                              void* low_a, void* low_g, cudaStream_t stream) {
    const DeltaDims dm{G, H, d, dv, taps, ra, rg};
    if (int rc = check_dims(dm)) return rc;
    AGV_REQUIRE(T >= 0 && B >= 0 && (row || part), "delta_prepare: no input");
    AGV_REQUIRE(state && conv_off >= (long long)H * dv * d &&
                state_stride >= conv_off + (long long)(taps - 1) * dm.C(),
                "delta_prepare: the state is too small");
    if (T == 0) return 0;
    const DeltaState st{state, state_stride, conv_off, slots, cu, seq_index, positions};
    // The rows form: a step of one token a sequence takes a token a warp, which alone has the warps to hide its
    // trips, others eight.  Those want whole lanes, since a head's channels have a warp to themselves: taken
    // for heads of up to 128 whose channels fill three quarters of the lanes, and enough channels or tokens
    // that the longer walk of a warp is hidden (or many channels and few tokens).  Against a CTA a token (us): 5,120 tokens, 16 heads of 128 213 and
    // 125, of 96 170 and 136, of 64 228 and 227, 8 of 64 118 and 128, 16 of 16 85 and 174, 4 of 256 213 and 229 (two
    // pieces a lane, too many registers); 300 tokens of 768 channels 14.6 and 16.3, 600 20.7 and 16.3, 300 of 2,304
    // 26.5 and 25.8, of 3,072 channels, heads of 64, 34.7 and 29.6.
    const int W = dm.W(), C = dm.C();
    const bool rows_can = (part || dtype == AGV_F32) && (part || ld % 4 == 0) && W % 4 == 0 && C % 4 == 0 && d % 4 == 0 &&
                          d <= (several ? 128 : 256) && taps >= 2 && taps <= 4 && state_stride % 4 == 0 &&
                          conv_off % 4 == 0 && agv_aligned(row, 16) && agv_aligned(part, 16) && agv_aligned(conv_w, 16) &&
                          agv_aligned(state, 16) && agv_aligned(qkv, 16);
    const long long lanes = 128LL * (2 * G + (dm.nv() + 127) / 128);
    const bool rows_pay = !several || (4LL * C >= 3 * lanes && (C >= 1536 || T >= 512)) ||
                          (5LL * C >= 3 * lanes && C >= 3072 && T <= 1024);
    AGV_REQUIRE(form >= 0 && form <= 2, "delta_prepare: no form %d", form);
    AGV_REQUIRE(form != 1 || rows_can, "delta_prepare: the rows form does not take these rows");
    if (form == 1 || (form == 0 && rows_can && rows_pay)) {
        AGV_REQUIRE(dtype == AGV_F32 || dtype == AGV_BF16, "delta_prepare: unknown dtype %d", dtype);
        const RowIn<float> in{(const float*)row, ld, part, n_splits, (long long)T * W, W};
        const int NJ = d <= 128 ? 1 : 2, R = several ? 8 : 1;
        const int n_seg = 2 * G + (dm.nv() + NJ * 128 - 1) / (NJ * 128) + (H + ra + rg + 31) / 32;
        const long long warps = (long long)((T + R - 1) / R) * n_seg;
        AGV_REQUIRE((warps + 3) / 4 <= 0x7fffffffLL, "delta_prepare: %d tokens exceed the grid limit", T);
        auto go = [&](auto kern, auto* la, auto* lg) {
            agv_launch(kern, (unsigned)((warps + 3) / 4), 128, 0, stream, in, dm, st, T, n_seg, conv_w, eps_unit,
                       q_mult, several ? 0 : 1, qkv, beta, la, lg);
        };
#define AGV_DPR(TT, TAPS) do {                                                                               \
        if (several) go(delta_prepare_rows_kernel<TT, TAPS, 1, 8>, (TT*)low_a, (TT*)low_g);                      \
        else if (NJ == 1) go(delta_prepare_rows_kernel<TT, TAPS, 1, 1>, (TT*)low_a, (TT*)low_g);                 \
        else go(delta_prepare_rows_kernel<TT, TAPS, 2, 1>, (TT*)low_a, (TT*)low_g); } while (0)
#define AGV_DPT(TT) do {                                                                                     \
        if (taps == 4) AGV_DPR(TT, 4); else if (taps == 3) AGV_DPR(TT, 3); else AGV_DPR(TT, 2); } while (0)
        if (dtype == AGV_F32) AGV_DPT(float); else AGV_DPT(__nv_bfloat16);
#undef AGV_DPT
#undef AGV_DPR
        AGV_LAUNCH_OK("delta_prepare_rows_kernel");
        if (several) {
            agv_launch(delta_conv_state_kernel<float>, (unsigned)B, 256, 0, stream, in, dm, st);
            AGV_LAUNCH_OK("delta_conv_state_kernel");
        }
        return 0;
    }
    const size_t smem = (size_t)(dm.C() + dm.W()) * sizeof(float);
#define AGV_DP(TT)                                                                              \
    do {                                                                                        \
        RowIn<TT> in{(const TT*)row, ld, part, n_splits, (long long)T * dm.W(), dm.W()};        \
        auto kern = delta_prepare_kernel<TT>;                                                   \
        if (smem > 48 * 1024)                                                                   \
            AGV_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                             (int)smem));                                       \
        agv_launch(kern, (unsigned)T, 256, smem, stream, in, dm, st, conv_w, eps_unit, q_mult,  \
                   several ? 0 : 1, qkv, beta, (TT*)low_a, (TT*)low_g);                         \
        AGV_LAUNCH_OK("delta_prepare_kernel");                                                  \
        if (several && taps > 1) {                                                              \
            agv_launch(delta_conv_state_kernel<TT>, (unsigned)B, 256, 0, stream, in, dm, st);   \
            AGV_LAUNCH_OK("delta_conv_state_kernel");                                           \
        }                                                                                       \
    } while (0)
    AGV_REQUIRE(smem <= 200 * 1024, "delta_prepare: %d channels exceed shared memory", dm.C());
    if (dtype == AGV_F32) AGV_DP(float);
    else if (dtype == AGV_BF16) AGV_DP(__nv_bfloat16);
    else return agv_fail(-1, "delta_prepare: unknown dtype %d", dtype);
#undef AGV_DP
    return 0;
}

// The recurrence over the step's tokens, sequence by sequence; all tensors 32-bit.
// work: scratch of agv_delta_scan_work(T, H, d) floats.
AGV_API long long agv_delta_scan_work(int T, int H, int d) {
    int L = 1;
    while (L * DL_R < d) L <<= 1;
    return (long long)T * H * (4LL * L * DL_R + 1);
}

AGV_API int agv_delta_scan(const float* qkv, const float* beta, const float* a,
                           const float* dt_bias, const float* neg_a, float* out, int T, int B,
                           int G, int H, int d, int dv, float* state, long long state_stride,
                           const int* slots, const int* cu, float* work, cudaStream_t stream) {
    const DeltaDims dm{G, H, d, dv, 1, 0, 0};
    if (int rc = check_dims(dm)) return rc;
    AGV_REQUIRE(state && state_stride >= (long long)H * dv * d, "delta_scan: the state is too small");
    AGV_REQUIRE(B <= 65535 && H <= 65535, "delta_scan: batch or head count exceeds the grid limit");
    if (T == 0 || B == 0) return 0;
    int L = 1;
    while (L * DL_R < d) L <<= 1;
    // 128 threads a CTA where the columns allow, whole warps always
    int CC = 128 / L;
    while (CC > 32 / L && CC / 2 >= dv) CC >>= 1;
    if (CC < 1) CC = 1;
    const int Dp = L * DL_R;
    // Two columns a lane where one would put more than two CTAs on every SM, in a step whose sequences
    // bring several tokens; a decode step is a read and a write of the state.
    const long long ctas = (long long)((dv + CC - 1) / CC) * H * B;
    const int CPT = T > B && dv >= 2 * CC && ctas > 296 ? 2 : 1;
    const int CW = CC * CPT;
    // two buffers of TCH tokens, within the 48 KB every launch may have
    int TCH = T <= B ? 1 : 16;             // (a decode step brings a token a sequence)
    while (TCH > 1 && 2 * scan_buf_floats(TCH, Dp, CW) * sizeof(float) > 46 * 1024) TCH >>= 1;
    const size_t smem = 2 * scan_buf_floats(TCH, Dp, CW) * sizeof(float);
    AGV_REQUIRE(smem <= 48 * 1024, "delta_scan: key heads of %d need too much shared memory", d);
    AGV_REQUIRE(work && ((size_t)work & 15) == 0, "delta_scan: no scratch, or not 16-byte aligned");
    const size_t row = (size_t)T * H * Dp;
    ScanArgs sa{qkv, beta, a, dt_bias, neg_a, out, L, CC, TCH,
                work, work + row, work + 2 * row, work + 3 * row, work + 4 * row};
    {
        const long long warps = (long long)T * H;
        agv_launch(delta_decay_kernel, (unsigned)((warps + 7) / 8), 256, 0, stream, sa, dm, T, Dp);
        AGV_LAUNCH_OK("delta_decay_kernel");
    }
    const DeltaState st{state, state_stride, 0, slots, cu, nullptr, nullptr};
    dim3 grid((unsigned)((dv + CW - 1) / CW), (unsigned)H, (unsigned)B);
    // (a STEP's tokens are a buffer each and its columns one a lane)
    auto go = [&](auto kern) { agv_launch_after(kern, grid, (unsigned)(CC * L), smem, stream, sa, dm, st); };
#define AGV_SCAN(LL)                                         \
    case LL:                                                 \
        if (T <= B) go(delta_scan_kernel<LL, 1, true>);      \
        else if (CPT == 1) go(delta_scan_kernel<LL, 1, false>); \
        else go(delta_scan_kernel<LL, 2, false>);            \
        break
    switch (L) {
        AGV_SCAN(1); AGV_SCAN(2); AGV_SCAN(4); AGV_SCAN(8); AGV_SCAN(16); AGV_SCAN(32);
        default: return agv_fail(-1, "delta_scan: %d lanes a column", L);
    }
#undef AGV_SCAN
    AGV_LAUNCH_OK("delta_scan_kernel");
    return 0;
}

// o, gate: [T, H * dv] 32-bit; w: [dv] 32-bit; y: [T, H * dv] in dtype.
AGV_API int agv_delta_out(const float* o, const float* gate, const float* w, float eps, int T,
                          int H, int dv, const int* seq_index, const int* slots, void* y,
                          int dtype, cudaStream_t stream) {
    AGV_REQUIRE(T >= 0 && H > 0 && dv > 0, "delta_out: bad sizes");
    if (T == 0) return 0;
    const bool four = dv % 4 == 0 && agv_aligned(o, 16) && agv_aligned(gate, 16) && agv_aligned(y, 8);
    const int L = dv <= 32 ? 8 : 32, heads = 128 / L;
    const long long grid = (long long)T * ((H + heads - 1) / heads);
    AGV_REQUIRE(grid <= 0x7fffffffLL, "delta_out: %d tokens exceed the grid limit", T);
#define AGV_DO(TT, VV, NN, LL) agv_launch(delta_out_kernel<TT, VV, NN, LL>, (unsigned)grid, 128, 0, stream, o, gate, w, \
                                          eps, T, H, dv, seq_index, slots, (TT*)y)
#define AGV_DOT(TT) do {                                                                \
        if (L == 8) { if (four) AGV_DO(TT, 4, 1, 8); else AGV_DO(TT, 1, 4, 8); }        \
        else if (dv <= 128) { if (four) AGV_DO(TT, 4, 1, 32); else AGV_DO(TT, 1, 4, 32); } \
        else { if (four) AGV_DO(TT, 4, 4, 32); else AGV_DO(TT, 1, 16, 32); } } while (0)
    if (dtype == AGV_F32) AGV_DOT(float);
    else if (dtype == AGV_BF16) AGV_DOT(__nv_bfloat16);
    else return agv_fail(-1, "delta_out: unknown dtype %d", dtype);
#undef AGV_DOT
#undef AGV_DO
    AGV_LAUNCH_OK("delta_out_kernel");
    return 0;
}
