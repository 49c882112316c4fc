"""Kernels that move a token's row four values or 16 bytes at a time, against their general forms
(which a weight off its 16-byte boundary selects), at the edges of their warps, tiles and pieces."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"
BF, F32 = torch.bfloat16, torch.float32


def rnd(*shape, dtype=F32, seed=0, scale=1.0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


def off(t):
    """The same values one element off a 16-byte boundary."""
    return torch.cat([t.reshape(-1)[:1], t.reshape(-1)])[1:].view(t.shape)


def same(a, b, dtype=F32):
    # (sums in another order: a few roundings of the largest value; bfloat16 results may fall on
    # either side of a rounding of 2^-9)
    tol = 3e-6 if dtype == F32 else 2.0 ** -8
    a, b = a.double(), b.double()
    assert torch.isfinite(a).all()
    assert float((a - b).abs().max()) <= tol * float(b.abs().max().clamp_min(1e-30))


def step(counts, starts, slots):
    i = dict(dtype=torch.int32, device=DEV)
    cu = [0]
    for n in counts:
        cu.append(cu[-1] + n)
    return SimpleNamespace(
        batch=len(counts), mode="decode" if max(counts) == 1 else "prefill",
        cu_seqlens=torch.tensor(cu, **i), slots=torch.tensor(slots, **i),
        seq_index=torch.tensor([b for b, n in enumerate(counts) for _ in range(n)], **i),
        positions=torch.tensor([s + k for s, n in zip(starts, counts) for k in range(n)], **i))


@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("G,H,d,dv,splits,dtype", [(2, 4, 128, 128, 3, BF), (1, 3, 36, 20, 1, BF),
                                                   (2, 2, 256, 200, 1, F32), (3, 3, 132, 4, 2, F32)])
@pytest.mark.parametrize("counts,starts", [([1, 1, 1], [5, 0, 2]), ([17, 1, 30], [0, 0, 0]),
                                           ([9, 3, 2], [4, 1, 0])])
def test_delta_prepare_rows(taps, G, H, d, dv, splits, dtype, counts, starts):
    """One token a warp and eight, sequences that begin and end inside a tile or go on from the
    ring, a padding entry."""
    from agave_b200 import kernels
    T, ra, rg = sum(counts), 8, 12
    C = 2 * G * d + H * dv
    W = (C + H + ra + rg + 3) // 4 * 4
    ra += W - (C + H + ra + rg)
    ctx = step(counts, starts, [2, -1, 0] if max(counts) == 1 else [2, 1, 0])
    part = rnd(splits, T, W, seed=1)
    conv_w = rnd(C, taps, seed=2, scale=0.5)
    off0 = H * dv * d + (-H * dv * d) % 4
    state0 = rnd(3, off0 + (taps - 1) * C, seed=3)
    outs = []
    for w, form in ((conv_w, "token"), (off(conv_w), "auto"), (conv_w, "rows"), (conv_w, "auto")):
        if form == "rows" and d > 128 and ctx.mode != "decode":
            with pytest.raises(kernels.KernelError, match="rows form"):
                kernels.delta_prepare(None, part, T, ctx, state0.clone(), off0, G, H, d, dv, taps, ra, rg, w, 1e-6,
                                      0.3, qkv, beta, la, lg, form=form)
            continue
        state = state0.clone()
        qkv, beta = torch.zeros(T, C, device=DEV), torch.zeros(T, H, device=DEV)
        la, lg = (torch.zeros(T, r, dtype=dtype, device=DEV) for r in (ra, rg))
        kernels.delta_prepare(None, part, T, ctx, state, off0, G, H, d, dv, taps, ra, rg, w, 1e-6,
                              0.3, qkv, beta, la, lg, form=form)
        outs.append((qkv, beta, la, lg, state))
    for got in outs[1:]:
        for a, b in zip(outs[0], got):
            same(b, a)


@pytest.mark.parametrize("taps", [2, 4])
@pytest.mark.parametrize("starts", [0, 3])
def test_delta_prepare_of_steps_one_after_the_other(taps, starts):
    """Steps that follow each other with no other kernel between them, a prompt and then single tokens,
    recorded together: each finds in the ring what the one before wrote there."""
    from agave_b200 import kernels
    G, H, d, dv, ra, rg, B, N = 2, 4, 128, 64, 8, 12, 3, 9
    C = 2 * G * d + H * dv
    W = C + H + ra + rg
    rows, conv_w = rnd(1, B * (7 + N), W, seed=1), rnd(C, taps, seed=2, scale=0.5)
    off0 = H * dv * d
    state0 = rnd(B, off0 + (taps - 1) * C, seed=3)
    part = rows.view(B, 7 + N, W)
    steps = [(step([7] * B, [starts] * B, list(range(B))), part[:, :7].reshape(1, B * 7, W).contiguous())]
    steps += [(step([1] * B, [starts + 7 + i] * B, list(range(B))), part[:, 7 + i].reshape(1, B, W).contiguous())
              for i in range(N)]
    outs = [(torch.zeros(x.shape[1], C, device=DEV), torch.zeros(x.shape[1], H, device=DEV),
             torch.zeros(x.shape[1], ra, device=DEV), torch.zeros(x.shape[1], rg, device=DEV)) for _, x in steps]

    def run(state):
        for (ctx, x), o in zip(steps, outs):
            kernels.delta_prepare(None, x, x.shape[1], ctx, state, off0, G, H, d, dv, taps, ra, rg, conv_w, 1e-6,
                                  0.3, *o, form="rows")
    state = state0.clone()
    run(state)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(state)
    # all tokens in one step
    whole = torch.zeros(B * (7 + N), C, device=DEV)
    kernels.delta_prepare(None, rows, B * (7 + N), step([7 + N] * B, [starts] * B, list(range(B))), state0.clone(), off0,
                          G, H, d, dv, taps, ra, rg, conv_w, 1e-6, 0.3, whole, torch.zeros(B * (7 + N), H, device=DEV),
                          torch.zeros(B * (7 + N), ra, device=DEV), torch.zeros(B * (7 + N), rg, device=DEV),
                          form="token")
    for _ in range(20):
        state.copy_(state0)
        graph.replay()
        got = torch.cat([outs[0][0].view(B, 7, C)] + [o[0].view(B, 1, C) for o in outs[1:]], 1)
        same(got, whole.view(B, 7 + N, C))


@pytest.mark.parametrize("G,H,d,dv,counts", [
    (4, 16, 128, 128, [70, 1, 0, 33, 17]),              # two columns a lane: 2, 8 and 16 lanes a column,
    (2, 16, 128, 36, [5, 40, 1, 9, 18, 2, 33, 16]),     # last groups of columns that are not whole,
    (16, 48, 20, 130, [20] * 5), (1, 24, 256, 68, [3, 21, 34, 2]),
    (4, 16, 128, 100, [2] * 140),                       # more sequences than a CTA has threads to rank
    (2, 4, 64, 40, [50, 1, 20]), (3, 3, 500, 12, [18, 3]), (1, 2, 8, 3, [40]),      # one column
    (4, 16, 128, 128, [1] * 9), (2, 4, 300, 70, [1, 1])])                           # one token a sequence
def test_delta_scan(G, H, d, dv, counts):
    """Against the recurrence in 64 bits, with a padding entry, and bit for bit what the same form
    gives in another order of the sequences; the sequences one by one take one column a lane."""
    from agave_b200 import kernels
    T, B, C = sum(counts), len(counts), 2 * G * d + H * dv
    qkv = rnd(T, C, seed=1)
    for h in range(2 * G):                              # (q and k are unit vectors)
        qkv[:, h * d:(h + 1) * d] /= qkv[:, h * d:(h + 1) * d].norm(dim=1, keepdim=True)
    beta, a = torch.sigmoid(rnd(T, H, seed=2)), rnd(T, H * d, seed=3)
    bias, neg_a = rnd(H * d, seed=4), -torch.exp(rnd(H, seed=5) - 1.0)
    state0 = rnd(B + 1, H * dv * d + 4, seed=6)
    slots = [B - b for b in range(B)]
    pad = 1 if B > 2 else None
    if pad is not None:
        slots[pad] = -1

    def run(counts, rows, slots, state):
        ctx = step(counts, [0] * len(counts), slots)
        ctx.new = lambda *s, dtype: torch.empty(s, dtype=dtype, device=DEV)
        out = torch.full((len(rows), H * dv), float("nan"), device=DEV)
        kernels.delta_scan(qkv[rows].contiguous(), beta[rows].contiguous(), a[rows].contiguous(), bias, neg_a, out,
                           ctx, state, G, H, d, dv)
        return out
    state = state0.clone()
    every = torch.arange(T, device=DEV)
    out = run(counts, every, slots, state)
    # in 64 bits
    g = torch.exp(neg_a.double()[:, None] * torch.nn.functional.softplus((a + bias).double().view(T, H, d), threshold=1e9))
    q, k = (t.double().view(T, G, d).repeat_interleave(H // G, 1) for t in (qkv[:, :G * d], qkv[:, G * d:2 * G * d]))
    v = qkv[:, 2 * G * d:].double().view(T, H, dv)
    want, ends = torch.zeros(T, H, dv, dtype=torch.float64, device=DEV), state0.double()
    cuts = [sum(counts[:b]) for b in range(B + 1)]
    for b in range(B):
        if slots[b] < 0:
            continue
        S = state0[slots[b], :H * dv * d].double().view(H, dv, d)
        for t in range(cuts[b], cuts[b + 1]):
            S = S * g[t][:, None, :]
            u = beta[t].double()[:, None] * (v[t] - torch.einsum("hvd,hd->hv", S, k[t]))
            S = S + u[:, :, None] * k[t][:, None, :]
            want[t] = torch.einsum("hvd,hd->hv", S, q[t])
        ends[slots[b], :H * dv * d] = S.reshape(-1)
    live = torch.cat([torch.arange(cuts[b], cuts[b + 1], device=DEV) for b in range(B) if slots[b] >= 0])
    assert float((out.double().view(T, H, dv) - want)[live].norm() / want[live].norm()) < 2e-6
    assert float((state.double() - ends).norm() / ends.norm()) < 2e-6
    assert torch.equal(state[:, H * dv * d:], state0[:, H * dv * d:]) and torch.equal(state[0], state0[0])
    # the sequences in reverse
    order = [b for b in range(B)][::-1]
    again = state0.clone()
    rows = torch.cat([every[cuts[b]:cuts[b + 1]] for b in order])
    back = run([counts[b] for b in order], rows, [slots[b] for b in order], again)
    keep = torch.isin(rows, live)
    assert torch.equal(back[keep], out[rows[keep]]) and torch.equal(again, state)
    # one by one: the same numbers but for the order of a column's sums
    for b in range(min(B, 8)):
        if slots[b] >= 0 and counts[b]:
            own = every[cuts[b]:cuts[b + 1]]
            same(run([counts[b]], own, [slots[b]], state0.clone()), out[own])


@pytest.mark.parametrize("T,H,dv", [(1, 3, 128), (9, 16, 128), (5, 2, 516), (4, 1, 700), (130, 3, 4)])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_delta_out_by_fours(T, H, dv, dtype):
    from agave_b200 import kernels
    ctx = step([1] * T, [1] * T, [-1 if t == 3 else t for t in range(T)])
    o, gate, w = rnd(T, H * dv, seed=1), rnd(T, H * dv, seed=2), rnd(dv, seed=3)
    ys = []
    for g in (gate, off(gate)):
        y = torch.full((T, H * dv), float("nan"), dtype=dtype, device=DEV)
        kernels.delta_out(o, g, w, 1e-6, H, dv, ctx, y)
        ys.append(y)
    same(*ys, dtype)
    if T > 3:
        assert not ys[0][3].any()


@pytest.mark.parametrize("T,H,dv", [(5, 3, 4), (7, 17, 20), (3, 16, 32), (6, 5, 33), (9, 33, 30), (2, 2, 132), (4, 3, 513),
                                     (2000, 5, 16)])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_delta_out(T, H, dv, dtype):
    """Eight lanes a head and a warp a head, heads that fill no CTA, columns kept and read again, in fours and
    one by one, in 64 bits; a padding entry's row."""
    from agave_b200 import kernels
    ctx = step([1] * T, [1] * T, [-1 if t == 2 else t for t in range(T)])
    o, gate, w = rnd(T, H * dv, seed=1), rnd(T, H * dv, seed=2), rnd(dv, seed=3)
    x = o.double().view(T, H, dv)
    want = (x / torch.sqrt((x * x).mean(-1, keepdim=True) + 1e-6) * w.double()).view(T, -1) * torch.sigmoid(gate.double())
    if T > 2:
        want[2] = 0.0
    for g in (gate, off(gate)):
        y = torch.full((T, H * dv), float("nan"), dtype=dtype, device=DEV)
        kernels.delta_out(o, g, w, 1e-6, H, dv, ctx, y)
        same(y, want, dtype)


@pytest.mark.parametrize("H,R,S", [(256, 70, 1), (512, 300, 2), (1000, 65, 1), (1028, 65, 2), (1028, 1024, 1), (1152, 1024, 2),
                                   (1152, 1025, 1), (1536, 1025, 2), (1540, 1025, 1), (2048, 65, 2), (2048, 1025, 1),
                                   (2560, 70, 2), (5000, 66, 1)])
@pytest.mark.parametrize("rms", [False, True])
def test_layer_norm_of_prompts(H, R, S, rms):
    """A warp a row and a CTA a row on both sides of every size at which they change places, the stream's row asked
    for early and late: branch norm, multiplier, residual sum and next norm in 64 bits."""
    from agave_b200 import kernels
    h, y = rnd(R, H, seed=1), rnd(S, R, H, seed=2)
    w1, b1, w2, b2 = (rnd(H, seed=3 + i) for i in range(4))

    def norm(v, w, b, eps):
        c = v if rms else v - v.mean(-1, keepdim=True)
        return c / torch.sqrt((c * c).mean(-1, keepdim=True) + eps) * w.double() + b.double()
    got, x = h.clone(), torch.empty(R, H, device=DEV)
    kernels.layer_norm_join(got, y, w1, b1, w2, b2, x, eps_post=1e-5, eps_next=1e-6, mult=0.7, rms=rms)
    want = h.double() + 0.7 * norm(y.double().sum(0), w1, b1, 1e-5)
    same(got, want)
    same(x, norm(want, w2, b2, 1e-6))


@pytest.mark.parametrize("T,K,H", [(1, 8, 4), (9, 2048, 2048), (3, 2056, 2052), (2, 4104, 4100)])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_row_gate_by_pieces(T, K, H, dtype):
    from agave_b200 import kernels
    x, w, y0 = rnd(T, K, dtype=dtype, seed=1), rnd(K, dtype=dtype, seed=2, scale=0.05), rnd(T, H, seed=3)
    ys = []
    for v in (w, off(w)):
        y = y0.clone()
        kernels.row_gate(x, v, y)
        ys.append(y)
    same(*ys)


@pytest.mark.parametrize("T,H,E,top", [(1, 8, 4, 2), (64, 2048, 32, 4), (3, 2056, 33, 3), (5, 4616, 70, 6),
                                       (64, 1024, 17, 2), (65, 1024, 17, 2), (3, 1024, 16, 2), (3, 1016, 17, 2),
                                       (3, 512, 40, 2), (3, 508 * 2, 200, 5)])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_route_of_few_tokens(T, H, E, top, dtype):
    """A warp an expert: one round of experts and several, rows of one round of pieces and more; the sizes at
    which sixteen warps and shared CTAs take over."""
    from agave_b200 import kernels
    x, w = rnd(T, H, dtype=dtype, seed=1), rnd(E, H, dtype=dtype, seed=2, scale=0.05)
    got = []
    for v in (w, off(w)):
        ids = torch.empty(T, top, dtype=torch.int32, device=DEV)
        wts = torch.empty(T, top, device=DEV)
        kernels.moe_route(x, v, None, 1, 1, top, ids, wts, softmax_top=True)
        got.append((ids, wts))
    assert torch.equal(got[0][0], got[1][0])
    same(got[0][1], got[1][1])


@pytest.mark.parametrize("T", [3, 70])
@pytest.mark.parametrize("nq,nk,nv,splits", [(4, 4, 4, 1), (2048, 512, 512, 3), (260, 516, 8, 2), (4000, 2000, 1004, 1)])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_proj_norm_by_fours(T, nq, nk, nv, splits, dtype):
    from agave_b200 import kernels
    part = rnd(splits, T, nq + nk + nv, seed=1)
    wq, wk, vf = rnd(nq, seed=2), rnd(nk, seed=3), rnd(T, nv, dtype=dtype, seed=4)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    for first in (None, vf):
        outs = []
        for w in (wq, off(wq)):
            out = torch.full((T, nq + nk + nv), float("nan"), dtype=dtype, device=DEV)
            kernels.proj_norm_store(out, nq, nk, nv, w, wk, 1e-6, pos, partial=part, v_first=first, v_mix=0.3)
            outs.append(out)
        same(*outs, dtype)


@pytest.mark.parametrize("T", [3, 70])
@pytest.mark.parametrize("latent", [False, True])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("A,d,r,R,G", [(16, 128, 64, 192, 16), (3, 4, 8, 4, 0), (2, 20, 24, 36, 40)])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_latent_prepare_by_fours(T, latent, interleaved, A, d, r, R, G, dtype):
    from agave_b200 import kernels
    Q = 60 if latent else A * (d + r)
    part = rnd(2, T, Q + R + r + G, seed=1)
    wq, wc = (rnd(Q, seed=2) if latent else None), rnd(R, seed=3)
    cos, sin = rnd(T, r // 2, seed=4), rnd(T, r // 2, seed=5)
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    outs = []
    for w in (wc, off(wc)):
        out = torch.full((T, Q + R + r + G), float("nan"), dtype=dtype, device=DEV)
        kernels.latent_prepare(out, Q, latent, A, d, r, R, G, wq, w, 1e-6, cos, sin, interleaved, pos, partial=part)
        outs.append(out)
    same(*outs, dtype)


def paged(counts, slots, width, cap, dtype, page=4):
    """A cache of rings of `cap` rows in scattered pages, and the step that whole sequences of these lengths make."""
    ctx = step(counts, [0] * len(counts), slots)
    ctx.lens = torch.tensor(counts, dtype=torch.int32, device=DEV)
    per = cap // page
    g = torch.Generator().manual_seed(cap)
    table = torch.randperm(len(counts) * per, generator=g).int().view(len(counts), per).contiguous().to(DEV)
    pool = torch.full((len(counts) * per, page, 1, width), 7.0, dtype=dtype, device=DEV)
    return ctx, SimpleNamespace(k_pool=pool, v_pool=pool, page_table=table, page=page, cap=cap)


def in_cache(view, counts, slots, rows):
    """What the pool holds when each sequence's last `cap` rows are in their ring."""
    want, at = torch.full_like(view.k_pool, 7.0), 0
    for n, slot in zip(counts, slots):
        for p in range(max(0, n - view.cap), n):
            if slot >= 0:
                r = p % view.cap
                want[int(view.page_table[slot, r // view.page]), r % view.page, 0] = rows[at + p]
        at += n
    return want


@pytest.mark.parametrize("counts,slots", [([5, 1, 9], [2, 0, 1]), ([40, 3, 60], [1, -1, 0]), ([200, 90, 30], [0, 2, 1])])
@pytest.mark.parametrize("nq,nk,nv", [(64, 16, 16), (2048, 512, 512)])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_proj_norm_by_fours_into_the_cache(counts, slots, nq, nk, nv, dtype):
    """Keys and values of few and of many tokens into rings that keep a sequence's end, beside a padding entry."""
    from agave_b200 import kernels
    T = sum(counts)
    part, wq, wk = rnd(2, T, nq + nk + nv, seed=1), rnd(nq, seed=2), rnd(nk, seed=3)
    for w in (wq, off(wq)):
        ctx, view = paged(counts, slots, nk, 32, dtype)
        view.v_pool = torch.full((*view.k_pool.shape[:3], nv), 7.0, dtype=dtype, device=DEV)
        out = torch.full((T, nq + nk + nv), float("nan"), dtype=dtype, device=DEV)
        kernels.proj_norm_store(out, nq, nk, nv, w, wk, 1e-6, ctx.positions, view, ctx, partial=part)
        assert torch.equal(view.k_pool, in_cache(view, counts, slots, out[:, nq:nq + nk]))
        both = SimpleNamespace(**{**vars(view), "k_pool": view.v_pool})
        assert torch.equal(view.v_pool, in_cache(both, counts, slots, out[:, nq + nk:]))


@pytest.mark.parametrize("counts,slots", [([5, 1, 9], [2, 0, 1]), ([40, 3, 60], [1, -1, 0]), ([200, 90, 30], [0, 2, 1]),
                                          ([300, 100, 150], [2, 0, 1])])
@pytest.mark.parametrize("latent", [False, True])
@pytest.mark.parametrize("A,d,r,R,G", [(2, 20, 24, 36, 40), (16, 128, 64, 512, 16), (16, 64, 64, 192, 2048), (32, 128, 64, 512, 32)])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_latent_prepare_by_fours_into_the_cache(counts, slots, latent, A, d, r, R, G, dtype):
    """Latent and key part of few and of many tokens into rings, at the widths and row counts at which threads and
    forms change places: the same rows as the general form's."""
    from agave_b200 import kernels
    T, Q = sum(counts), 60 if latent else A * (d + r)
    part = rnd(1, T, Q + R + r + G, seed=1)
    wq, wc = (rnd(Q, seed=2) if latent else None), rnd(R, seed=3)
    cos, sin = rnd(T, r // 2, seed=4), rnd(T, r // 2, seed=5)
    outs = []
    for w in (wc, off(wc)):
        ctx, view = paged(counts, slots, R + r, 32, dtype)
        out = torch.full((T, Q + R + r + G), float("nan"), dtype=dtype, device=DEV)
        kernels.latent_prepare(out, Q, latent, A, d, r, R, G, wq, w, 1e-6, cos, sin, latent, ctx.positions, view, ctx,
                               partial=part)
        assert torch.equal(view.k_pool, in_cache(view, counts, slots, out[:, Q:Q + R + r]))
        outs.append(out)
    same(*outs, dtype)


@pytest.mark.parametrize("H,G,d,dv", [(4, 1, 128, 64), (2, 2, 64, 32), (3, 1, 200, 100), (2, 1, 256, 34)])
@pytest.mark.parametrize("counts", [[192], [1, 300, 64, 3], [129, 128, 127, 515]])
@pytest.mark.parametrize("strong", [False, True])
def test_head_scan_by_chunks(H, G, d, dv, counts, strong):
    """Chunks that end inside, at and after a sequence's end, states that go on from another step,
    decays near one and near (and at) zero: against the recurrence in 64 bits, no further from it than the
    scan token by token (with room for the order of the sums)."""
    from agave_b200 import kernels
    T, B, W = sum(counts), len(counts), 2 * G * d + H * dv + 4
    ctx = step(counts, [0] * B, list(range(B)))
    row = rnd(T, W, seed=1)
    q, k, v = row[:, :G * d], row[:, G * d:2 * G * d], row[:, 2 * G * d:2 * G * d + H * dv]
    a = torch.exp(-torch.exp(rnd(T, H, seed=2, scale=2.0) + (1.0 if strong else -5.0)))
    if strong:
        a[T // 2] = 0.0
    coef = torch.stack([a, rnd(T, H, seed=3).abs()], -1).contiguous()
    state0 = rnd(B, 5 + H * d * dv, seed=4)
    S = state0[:, 5:].view(B, H, d, dv).double()
    want = torch.empty(T, H, dv, dtype=torch.float64, device=DEV)
    q8, k8 = (t.double().view(T, G, d).repeat_interleave(H // G, 1) for t in (q, k))
    v8, c8 = v.double().view(T, H, dv), coef.double()
    at = 0
    for b, n in enumerate(counts):
        for t in range(at, at + n):
            S[b] = c8[t, :, 0, None, None] * S[b] + c8[t, :, 1, None, None] * k8[t, :, :, None] * v8[t, :, None]
            want[t] = torch.einsum("hd,hdv->hv", q8[t], S[b])
        at += n
    err = {}
    for form in ("tokens", "chunks"):
        state, out = state0.clone(), torch.full((T, H * dv), float("nan"), device=DEV)
        kernels.head_scan(q, k, v, coef, out, ctx, state, 5, H, G, d, dv, form=form)
        err[form] = [float((g.double() - r).norm() / r.norm()) for g, r in
                        ((out.view(T, H, dv), want), (state[:, 5:].view(B, H, d, dv), S))]
        assert torch.equal(state[:, :5], state0[:, :5])
    for token, chunk in zip(err["tokens"], err["chunks"]):
        assert chunk <= 1.5 * token + 1e-7 and chunk < 2e-6, err


@pytest.mark.parametrize("H,G,d,dv", [(2, 1, 64, 64), (3, 3, 200, 100)])
@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
def test_head_scan_values_reach_no_earlier_token(H, G, d, dv, bad):
    """A value that is infinite or NaN, at the first, a middle and the last token of a chunk's
    block of sixteen: every earlier token's output is bit for bit what it is without it, and its
    own and later ones in that column are not finite."""
    from agave_b200 import kernels
    T, W = 300, 2 * G * d + H * dv
    ctx = step([T], [0], [0])
    row = rnd(T, W, seed=1)
    coef = torch.stack([torch.sigmoid(rnd(T, H, seed=2) + 4.0), rnd(T, H, seed=3).abs() + 0.1], -1).contiguous()
    got = []
    for at in (None, 128, 137, 143, 255, 299):
        r = row.clone()
        if at is not None:
            r[at, 2 * G * d + 5] = bad                       # head 0, column 5
        q, k, v = r[:, :G * d], r[:, G * d:2 * G * d], r[:, 2 * G * d:]
        out = torch.empty(T, H * dv, device=DEV)
        kernels.head_scan(q, k, v, coef, out, ctx, torch.zeros(1, H * d * dv, device=DEV), 0, H, G, d, dv,
                          form="chunks")
        got.append(out)
        if at is not None:
            assert torch.equal(out[:at], got[0][:at]), at
            assert not torch.isfinite(out[at:, 5]).any()
            others = torch.arange(H * dv, device=DEV) != 5
            assert torch.equal(out[:, others], got[0][:, others])


@pytest.mark.parametrize("pad", [0, 1, 2])
@pytest.mark.parametrize("H,G,d,dv", [(2, 1, 64, 64), (3, 3, 200, 100)])
def test_head_scan_padding_entries_are_zeros(H, G, d, dv, pad):
    """A padding entry of a prompt step gets rows of zeros and touches no state, by chunks as token by
    token, and the other entries are bit for bit what they are without one."""
    from agave_b200 import kernels
    counts = [130, 400, 65]
    T, W = sum(counts), 2 * G * d + H * dv
    row = rnd(T, W, seed=1)
    q, k, v = row[:, :G * d], row[:, G * d:2 * G * d], row[:, 2 * G * d:]
    coef = torch.stack([torch.sigmoid(rnd(T, H, seed=2) + 2.0), rnd(T, H, seed=3).abs()], -1).contiguous()
    state0 = rnd(3, H * d * dv, seed=4)
    for form in ("tokens", "chunks"):
        got = []
        for s in ([0, 1, 2], [b if b != pad else -1 for b in range(3)]):
            ctx = step(counts, [0] * 3, s)
            state, out = state0.clone(), torch.full((T, H * dv), float("nan"), device=DEV)
            kernels.head_scan(q, k, v, coef, out, ctx, state, 0, H, G, d, dv, form=form)
            got.append((out, state))
        rows = torch.zeros(T, dtype=torch.bool, device=DEV)
        rows[sum(counts[:pad]):sum(counts[:pad + 1])] = True
        assert not got[1][0][rows].any()
        assert torch.equal(got[1][0][~rows], got[0][0][~rows])
        assert torch.equal(got[1][1][pad], state0[pad])
        keep = [b for b in range(3) if b != pad]
        assert torch.equal(got[1][1][keep], got[0][1][keep])


@pytest.mark.parametrize("inner,N", [(96, 16), (130, 4), (64, 7), (33, 128), (48, 200)])
@pytest.mark.parametrize("counts", [[150], [1, 700, 96, 3], [192, 191, 97, 515]])
@pytest.mark.parametrize("dtype", [BF, F32])
def test_selective_scan_by_segments(inner, N, counts, dtype):
    """Segments that end inside, at and after a sequence's end, states that go on from another step:
    against the scan of whole sequences (2^-21 a decay, over a segment once instead of a token)."""
    from agave_b200 import kernels
    T, B, Np = sum(counts), len(counts), kernels.selective_pad(N)
    ctx = step(counts, [0] * B, list(range(B)))
    u, dt, z = rnd(T, inner, seed=1), rnd(T, inner, seed=2) - 1.0, rnd(T, inner, seed=3)
    bc = torch.zeros(T, 2, Np, device=DEV)
    bc[:, :, :N] = rnd(T, 2, N, seed=4)
    a2 = -torch.exp(rnd(inner, N, seed=5, scale=2.0) - 2.0)
    bias, d, state0 = rnd(inner, seed=6), rnd(inner, seed=7), rnd(B, 3 + inner * N, seed=8)
    got = []
    for form in ("whole", "segments"):
        state, out = state0.clone(), torch.full((T, inner), float("nan"), dtype=dtype, device=DEV)
        kernels.selective_scan(u, dt, bias, bc.view(T, -1), a2, d, z, None, inner, 0, out, ctx, state, 3, form=form)
        got.append((out, state))
    assert float((got[0][1] - got[1][1]).abs().max()) <= 4e-6 * float(got[0][1].abs().max())
    assert torch.equal(got[0][1][:, :3], got[1][1][:, :3])
    tol = 4e-6 if dtype == F32 else 2.0 ** -8
    assert float((got[0][0].double() - got[1][0].double()).abs().max()) <= tol * float(got[0][0].abs().max())


def test_scans_run_without_room_for_scratch(monkeypatch):
    """Where the device has no room for the chunks' and the segments' states, the scans take the
    form that needs none: the results of a step that asks for none."""
    from agave_b200 import kernels
    counts = [900, 80]
    T, H, G, d, dv, inner, N = sum(counts), 2, 1, 64, 64, 128, 16
    row = rnd(T, 2 * G * d + H * dv, seed=1)
    q, k, v = row[:, :G * d], row[:, G * d:2 * G * d], row[:, 2 * G * d:]
    coef = torch.stack([torch.sigmoid(rnd(T, H, seed=2) + 2.0), rnd(T, H, seed=3).abs()], -1).contiguous()
    u, dt, z, bc = (rnd(T, n, seed=4 + i) for i, n in enumerate((inner, inner, inner, 2 * N)))
    a2, bias, D = -torch.exp(rnd(inner, N, seed=8)), rnd(inner, seed=9), rnd(inner, seed=10)
    lib, ctx = kernels.library(), step(counts, [0, 0], [0, 1])
    assert lib.agv_head_scan_work(T, 2, H, G, d, dv, max(counts)) > 0
    assert lib.agv_selective_scan_work(T, 2, inner, N, max(counts)) > 0

    def both(out, y, S, state):
        kernels.head_scan(q, k, v, coef, out, ctx, S, 0, H, G, d, dv)
        kernels.selective_scan(u, dt, bias, bc, a2, D, z, None, inner, 0, y, ctx, state, 0)
        return out, y, S, state
    fresh = [(torch.empty(T, H * dv, device=DEV), torch.empty(T, inner, device=DEV), torch.zeros(2, H * d * dv, device=DEV),
              torch.zeros(2, inner * N, device=DEV)) for _ in range(2)]
    ctx.max_new = 1
    want = both(*fresh[0])
    ctx.max_new = max(counts)

    def full(*a, **k):
        raise torch.OutOfMemoryError("no room")
    monkeypatch.setattr(torch, "empty", full)
    got = both(*fresh[1])
    monkeypatch.undo()
    for a, b in zip(got, want):
        assert torch.equal(a, b)


def test_scratch_of_the_scans_is_bounded():
    """Whatever the batch, the states, the heads and the lengths, chosen or asked for: at most 512 MB."""
    import ctypes
    from agave_b200 import kernels
    lib = kernels.library()
    lib.agv_head_scan_work.restype = lib.agv_selective_scan_work.restype = ctypes.c_longlong
    some = 0
    for B in (1, 8, 64, 1024):
        for longest in (150, 2000, 100000):
            T = longest + (B - 1) * 64
            for wide in (1, 8, 64):
                for lengths in (longest, 0):
                    n = lib.agv_selective_scan_work(T, B, 128 * wide, 256, lengths)
                    m = lib.agv_head_scan_work(T, B, 2 * wide, 1, 128, 64, lengths)
                    assert 0 <= n <= 1 << 27 and 0 <= m <= 1 << 27
                    some += (n > 0) + (m > 0)
    assert some > 20


# lengths, heads, groups, state, values: whether the chunks are the faster form (both measured)
@pytest.mark.parametrize("counts,H,G,d,dv,chunks", [
    ([333, 1501], 64, 1, 128, 64, True), ([1024], 24, 1, 128, 64, True), ([4096], 8, 1, 64, 32, True),
    ([1], 64, 1, 128, 64, False), ([192] * 16, 48, 1, 64, 64, False), ([256] * 32, 16, 16, 64, 64, False),
    ([64] * 255 + [192], 16, 16, 64, 64, False), ([128] * 32, 64, 1, 128, 64, False), ([192], 32, 1, 256, 128, False)])
def test_head_scan_rule(counts, H, G, d, dv, chunks):
    import ctypes
    from agave_b200 import kernels
    lib = kernels.library()
    lib.agv_head_scan_work.restype = ctypes.c_longlong
    assert (lib.agv_head_scan_work(sum(counts), len(counts), H, G, d, dv, max(counts)) > 0) == chunks


@pytest.mark.parametrize("counts,inner,N,segments", [
    ([333, 1501], 4096, 16, True), ([4096], 512, 16, True), ([1024] * 4, 128, 16, True), ([512], 1024, 4, True),
    ([1], 4096, 16, False), ([384] * 2, 4096, 16, False), ([20] * 500 + [400], 512, 16, False),
    ([150], 2048, 128, False), ([256] * 32, 512, 16, False), ([400] * 2, 8192, 16, False)])
def test_selective_scan_rule(counts, inner, N, segments):
    import ctypes
    from agave_b200 import kernels
    lib = kernels.library()
    lib.agv_selective_scan_work.restype = ctypes.c_longlong
    assert (lib.agv_selective_scan_work(sum(counts), len(counts), inner, N, max(counts)) > 0) == segments


@pytest.mark.parametrize("B", [1, 31, 32, 33, 97])
def test_scans_find_their_pieces_in_any_batch(B):
    """Empty, short and long sequences in batches around a warp's 32: chunks and segments against the
    forms that take every sequence by itself."""
    from agave_b200 import kernels
    g = torch.Generator().manual_seed(B)
    counts = torch.randint(0, 3, (B,), generator=g).mul_(97).tolist()
    counts[-1] = 300
    T, H, G, d, dv, inner, N = sum(counts), 2, 1, 64, 32, 64, 16
    ctx = step(counts, [0] * B, list(range(B)))
    row = rnd(T, 2 * G * d + H * dv, seed=1)
    q, k, v = row[:, :G * d], row[:, G * d:2 * G * d], row[:, 2 * G * d:]
    coef = torch.stack([torch.sigmoid(rnd(T, H, seed=2) + 2.0), rnd(T, H, seed=3).abs()], -1).contiguous()
    u, dt, z, bc = (rnd(T, n, seed=4 + i) for i, n in enumerate((inner, inner, inner, 2 * N)))
    a2, bias, D = -torch.exp(rnd(inner, N, seed=8)), rnd(inner, seed=9), rnd(inner, seed=10)
    S0, s0 = rnd(B, H * d * dv, seed=11), rnd(B, inner * N, seed=12)
    got = []
    for head, sel in (("tokens", "whole"), ("chunks", "segments")):
        S, s, out, y = S0.clone(), s0.clone(), torch.empty(T, H * dv, device=DEV), torch.empty(T, inner, device=DEV)
        kernels.head_scan(q, k, v, coef, out, ctx, S, 0, H, G, d, dv, form=head)
        kernels.selective_scan(u, dt, bias, bc, a2, D, z, None, inner, 0, y, ctx, s, 0, form=sel)
        got.append((out, S, y, s))
    for a, b in zip(*got):
        same(b, a)


@pytest.mark.parametrize("inner,N", [(96, 16), (66, 4), (33, 128), (20, 200)])
@pytest.mark.parametrize("counts", [[200], [1, 500, 96, 3], [192, 191]])
@pytest.mark.parametrize("strong", [False, True])
def test_selective_scan_in_64_bits(inner, N, counts, strong):
    """Both forms against the recurrence in 64 bits, states that go on from another step, a padding entry, decays near
    one and near zero: segments no further off than whole sequences (with room for the order of the sums)."""
    from agave_b200 import kernels
    T, B, Np = sum(counts), len(counts), kernels.selective_pad(N)
    slots = [b if b != 2 else -1 for b in range(B)]
    ctx = step(counts, [0] * B, slots)
    u, dt, z = rnd(T, inner, seed=1), rnd(T, inner, seed=2) - 1.0, rnd(T, inner, seed=3)
    bc = torch.zeros(T, 2, Np, device=DEV)
    bc[:, :, :N] = rnd(T, 2, N, seed=4)
    a2 = -torch.exp(rnd(inner, N, seed=5, scale=1.0) + (2.0 if strong else -4.0))
    bias, d, state0 = rnd(inner, seed=6), rnd(inner, seed=7), rnd(B, 3 + inner * N, seed=8)
    step8 = torch.nn.functional.softplus((dt + bias).double(), threshold=1e9)
    want, ends, at = torch.zeros(T, inner, dtype=torch.float64, device=DEV), state0.double(), 0
    for b, n in enumerate(counts):
        S = state0[b, 3:].double().view(inner, N)
        for t in range(at, at + n):
            S = torch.exp2(step8[t][:, None] * a2.double()) * S + (step8[t] * u[t].double())[:, None] * bc[t, 0, :N].double()
            want[t] = S @ bc[t, 1, :N].double() + d.double() * u[t].double()
        if slots[b] >= 0:
            ends[b, 3:] = S.reshape(-1)
        else:
            want[at:at + n] = 0.0
        at += n
    want = want * torch.nn.functional.silu(z.double())
    err = {}
    for form in ("whole", "segments"):
        state, out = state0.clone(), torch.full((T, inner), float("nan"), device=DEV)
        kernels.selective_scan(u, dt, bias, bc.view(T, -1), a2, d, z, None, inner, 0, out, ctx, state, 3, form=form)
        err[form] = [float((g.double() - r).norm() / r.norm()) for g, r in ((out, want), (state, ends))]
        assert torch.equal(state[:, :3], state0[:, :3])
        if B > 2:
            assert torch.equal(state[2], state0[2])
    # (2^-22 a decay by the hardware's power of two, once a token, over states of some hundred tokens)
    for whole, cut in zip(err["whole"], err["segments"]):
        assert cut <= 1.5 * whole + 2e-7 and cut < 5e-6, err
