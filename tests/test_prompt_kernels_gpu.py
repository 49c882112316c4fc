"""Prompt kernels at the edges of their tiles, against sums written out in torch."""
import pytest
import torch

pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def rnd(*shape, dtype=torch.float32, seed=0, scale=1.0):
    g = torch.Generator(device="cpu").manual_seed(seed)
    return (torch.randn(*shape, generator=g) * scale).to(dtype).to(DEV)


def rel_err(got, ref):
    got, ref = got.double().cpu(), ref.double().cpu()
    return ((got - ref).abs().max() / ref.abs().max().clamp_min(1e-30)).item()


@pytest.mark.parametrize("nh,nkv,hd,hdv,window,keep", [
    (4, 1, 256, 256, 0, 0), (4, 1, 256, 256, 130, 0), (8, 4, 128, 128, 65, 0),
    (3, 3, 64, 192, 0, 0), (2, 1, 192, 48, 64, 0), (16, 1, 80, 144, 70, 5), (4, 2, 128, 128, 40, 130),
    (2, 2, 16, 16, 1, 0)])
def test_prompt_attention_at_the_edges_of_its_tiles(nh, nkv, hd, hdv, window, keep):
    """Lengths round half tiles of 64 keys and tiles of 128, an odd number of halves, windows that
    start inside one, kept first keys apart from the window, value heads of their own size (one
    and two slots a tile).  Errors: P, the values and the result are bfloat16 (2^-9 each)."""
    from agave_b200 import kernels
    lens = [1, 63, 64, 65, 127, 128, 129, 191, 192, 193, 256, 257, 321]
    T = sum(lens)
    q, k = (rnd(T, n * hd, dtype=torch.bfloat16, seed=i, scale=0.5) for i, n in enumerate((nh, nkv)))
    v = rnd(T, nkv * hdv, dtype=torch.bfloat16, seed=3)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    out = torch.full((T, nh * hdv), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.attention_prefill_tc(q, k, v, out, cu, max(lens), nh, nkv, hd, 0.3, window,
                                 value_dim=hdv, keep_first=keep)
    assert kernels.attention_tc_status() == 0
    o = 0
    for n in lens:
        at = slice(o, o + n)
        qs = q[at].double().reshape(n, nh, hd).transpose(0, 1)
        ks = k[at].double().reshape(n, nkv, hd).transpose(0, 1).repeat_interleave(nh // nkv, 0)
        vs = v[at].double().reshape(n, nkv, hdv).transpose(0, 1).repeat_interleave(nh // nkv, 0)
        p = torch.arange(n, device=DEV)[:, None]
        j = torch.arange(n, device=DEV)[None, :]
        see = (j <= p) & ((j > p - window) | (j < keep) if window else j >= 0)
        s = ((qs @ ks.transpose(1, 2)) * 0.3).masked_fill(~see, float("-inf"))
        ref = (torch.softmax(s, -1) @ vs).transpose(0, 1).reshape(n, nh * hdv)
        assert rel_err(out[at], ref) < 6e-3, n
        o += n


@pytest.mark.parametrize("T", [65, 100, 128])
@pytest.mark.parametrize("N,K", [(6912, 1152), (100, 72), (10240, 320), (4800, 64)])
def test_gated_product_of_short_prompts(T, N, K):
    """One or two tiles of features a CTA, a last tile that is not full, fewer and more k-blocks
    than stages.  The result is rounded to bfloat16 (2^-9), the gate's tanh is within 2^-11."""
    from agave_b200 import kernels
    x = rnd(T, K, dtype=torch.bfloat16, seed=7)
    wg, wu = (rnd(N, K, dtype=torch.bfloat16, seed=s, scale=K ** -0.5) for s in (8, 9))
    out = torch.full((T + 1, N + 8), float("nan"), dtype=torch.bfloat16, device=DEV)
    kernels.linear_tc(x, wg, out[:T, :N], w2=wu, activation="gelu_tanh")
    assert kernels.linear_tc_status() == 0
    ref = torch.nn.functional.gelu(x.double() @ wg.double().T, approximate="tanh") * (x.double() @ wu.double().T)
    assert rel_err(out[:T, :N], ref) < 6e-3
    assert torch.isnan(out[T]).all() and torch.isnan(out[:, N:]).all()


@pytest.mark.parametrize("T,N,K,splits,act", [
    (129, 130, 8192, 1, None), (300, 1150, 1096, 1, "relu2"), (2051, 2300, 2056, 1, "gelu_erf"),
    (3000, 1541, 4104, 1, None), (5000, 4100, 1032, 1, "relu2"), (4100, 1000, 1160, 2, None)])
def test_products_of_prompts_on_pairs_of_ctas(T, N, K, splits, act):
    """Tiles of 256, 192 and 128 features a pair: tokens and features that end inside a tile, rows
    whose stride is no multiple of four values, one and many rounds, K in two ranges and with a
    ragged end.  32-bit sums of bfloat16 products: errors of a sum of K terms in 32 bits."""
    from agave_b200 import kernels
    x = rnd(T, K, dtype=torch.bfloat16, seed=1)
    w = rnd(N, K, dtype=torch.bfloat16, seed=2, scale=K ** -0.5)
    ref = x.double() @ w.double().T
    for ld in (N + (-N) % 4, N + (-N) % 4 + 3):
        if splits > 1 and ld != N:
            continue
        out = torch.full((splits, T, ld) if splits > 1 else (T + 1, ld), float("nan"), device=DEV)
        kernels.linear_tc(x, w, out if splits > 1 else out[:T, :N], splits=splits)
        assert kernels.linear_tc_status() == 0
        assert rel_err(out.double().sum(0) if splits > 1 else out[:T, :N], ref) < 1e-5
        assert splits > 1 or (torch.isnan(out[T]).all() and torch.isnan(out[:, N:]).all())
    if act:
        ob = torch.full((T, N + 4 + (-N) % 4), float("nan"), dtype=torch.bfloat16, device=DEV)
        kernels.linear_activated(x, w, ob[:, :N], act)
        assert kernels.linear_tc_status() == 0
        want = torch.relu(ref) ** 2 if act == "relu2" else torch.nn.functional.gelu(ref)
        assert rel_err(ob[:, :N], want) < 6e-3 and torch.isnan(ob[:, N:]).all()


@pytest.mark.parametrize("nkv,hd", [(1, 256), (3, 64), (2, 192)])
@pytest.mark.parametrize("splits", [2, 8, 9, 16])
def test_transposed_values_of_short_prompts(nkv, hd, splits):
    """The values from several partial sums, transposed: sequences that end inside a tile of 64
    tokens or fill it, sums up to a batch of loads and beyond.  The sums are added in order in 32
    bits and rounded once, so they are what torch gives bit for bit."""
    from agave_b200 import kernels
    nh, lens = nkv, [64, 1, 37, 63, 65]
    T, W = sum(lens), (nh + 2 * nkv) * hd
    part = rnd(splits, T, W, seed=4)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(n) for n in lens]).int().to(DEV)
    seq = torch.cat([torch.full((n,), b) for b, n in enumerate(lens)]).int().to(DEV)
    cols = [(n + 63) // 64 * 64 for n in lens]
    vt = torch.full((nkv * hd, sum(cols) + 64), 7.0, dtype=torch.bfloat16, device=DEV)
    qkv = torch.empty(T, W, dtype=torch.bfloat16, device=DEV)
    kernels.qk_norm_rope_store(qkv, nh, nkv, hd, None, None, 1e-6, None, None, 0, pos, seq_index=seq,
                               partial=part, vt=vt, cu_seqlens=cu, max_len=max(lens))
    total = part[0].clone()
    for s in range(1, splits):
        total += part[s]
    v = total.to(torch.bfloat16)
    assert torch.equal(qkv, v)
    at = o = 0
    for n, c in zip(lens, cols):
        assert torch.equal(vt[:, at:at + n], v[o:o + n, (nh + nkv) * hd:].T), n
        assert not vt[:, at + n:at + c].any(), n
        at, o = at + c, o + n
    assert (vt[:, at:] == 7.0).all()


@pytest.mark.parametrize("N,K", [(1152, 1024), (2048, 1152), (2080, 1152), (40, 2312), (2016, 6920)])
@pytest.mark.parametrize("M", [1, 3, 4, 5])
def test_32_bit_products_either_side_of_the_deep_rings(N, K, M):
    """Weights of up to 64 groups of 32 rows and of more, walks shorter than a ring and with a ragged
    last piece, more rows than a deep ring takes.  A row's sum has one order whatever its company."""
    from agave_b200 import kernels
    x, w = rnd(M, K, seed=1), rnd(N, K, seed=2, scale=K ** -0.5)
    out = torch.full((M + 1, N), float("nan"), device=DEV)
    kernels.linear_simt(x, w, out[:M])
    ref = x.double() @ w.double().T
    assert rel_err(out[:M], ref) < 1e-6 and torch.isnan(out[M]).all()
    one = torch.empty(1, N, device=DEV)
    kernels.linear_simt(x[:1], w, one)
    assert torch.equal(one[0], out[0])


@pytest.mark.parametrize("tile", [64, 128])
@pytest.mark.parametrize("weigh_input", [False, True])
@pytest.mark.parametrize("T,E,top,H,ff", [(9, 6, 3, 264, 200), (3, 40, 4, 64, 136), (300, 5, 2, 136, 264),
                                          (1500, 7, 4, 1032, 72)])
def test_padding_of_the_experts_rows_reaches_nothing(tile, weigh_input, T, E, top, H, ff):
    """The plan's padding rows hold NaN before the rows are gathered and before both products: results
    are finite and right, the padding is as it was; one expert has no tokens and some choices name no
    expert at all.  A CTA a row, and pieces of rows that end inside a CTA.  z is rounded to bfloat16 (2^-9),
    its gate is within 2^-11 and sums are in 32 bits."""
    from agave_b200 import kernels
    g = torch.Generator().manual_seed(T + E)
    ids = torch.stack([torch.randperm(E + 2, generator=g)[:top] for _ in range(T)])
    ids[ids == 1] = E                                  # (nobody goes to expert 1)
    ids = ids.int().to(DEV)
    wts = torch.rand(T, top, generator=g).to(DEV) + 0.1
    x = rnd(T, H + 8, dtype=torch.bfloat16, seed=1)[:, :H]
    wg, wu = (rnd(E, ff, H, dtype=torch.bfloat16, seed=s, scale=H ** -0.5) for s in (2, 3))
    wd = rnd(E, H, ff, dtype=torch.bfloat16, seed=4, scale=ff ** -0.5)
    plan = kernels.moe_plan(ids, wts, E, tile=tile)
    nan = float("nan")
    xs = torch.full((plan.rows, H), nan, dtype=torch.bfloat16, device=DEV)
    z = torch.full((plan.rows, ff), nan, dtype=torch.bfloat16, device=DEV)
    y = torch.full((top * T, H), nan, device=DEV)
    kernels.moe_gather_rows(x, plan, xs)
    kernels.moe_grouped_tc(xs, wg, z, plan, w2=wu, activation="silu", weigh=weigh_input)
    kernels.moe_grouped_tc(z, wd, y, plan, scatter=True, weigh=not weigh_input)
    assert kernels.moe_tc_status() == 0
    pos = plan.pos_of.view(T, top).long()
    assert torch.equal(pos < 0, ids >= E)
    live = pos[pos >= 0]
    padding = torch.ones(plan.rows, dtype=torch.bool, device=DEV)
    padding[live] = False
    assert padding.any()
    for t in (xs, z):
        assert torch.isnan(t[padding]).all() and torch.isfinite(t[live]).all()
    want = torch.full((top, T, H), nan, dtype=torch.float64, device=DEV)
    for e in range(E):
        t, c = (ids == e).nonzero(as_tuple=True)
        if not len(t):
            continue
        assert torch.equal(xs[pos[t, c]], x[t])
        w = wts[t, c].double()[:, None]
        u, v = x[t].double() @ wg[e].double().T, x[t].double() @ wu[e].double().T
        if weigh_input:
            u, v = u * w, v * w
        r = (torch.nn.functional.silu(u) * v) @ wd[e].double().T
        want[c, t] = r if weigh_input else r * w
    got = y.view(top, T, H)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    there = ~torch.isnan(want)
    assert rel_err(got[there], want[there]) < 8e-3


@pytest.mark.parametrize("R", [192, 193, 444, 445])
@pytest.mark.parametrize("H,S", [(512, 5), (1024, 1), (1152, 3), (2048, 5), (2560, 4)])
def test_norm_with_its_weights_early_or_late(H, S, R):
    """Rows either side of the lines at which the weights are asked for before the wait.  Sums of S
    values and of H squares in 32 bits; the stream in 32 bits, the result rounded to bfloat16 (2^-9)."""
    from agave_b200 import kernels
    h0, y = rnd(R, H, seed=1), rnd(S, R, H, seed=2)
    wp, wn = 1 + rnd(H, seed=3, scale=0.1), 1 + rnd(H, seed=4, scale=0.1)
    h, x = h0.clone(), torch.empty(R, H, dtype=torch.bfloat16, device=DEV)
    kernels.norm_residual(h, y if S > 1 else y[0], wp, wn, x, 1e-6, 1e-6)
    b = y.double().sum(0)
    want = h0.double() + b / (b.square().mean(1, keepdim=True) + 1e-6).sqrt() * wp.double()
    assert rel_err(h, want) < 2e-6
    assert rel_err(x, want / (want.square().mean(1, keepdim=True) + 1e-6).sqrt() * wn.double()) < 4e-3


@pytest.mark.parametrize("splits", [1, 2, 9])
@pytest.mark.parametrize("nh,nkv,hd,lens", [
    (8, 4, 64, [64, 1, 700, 63, 513, 128]), (3, 1, 256, [1200, 70]), (5, 2, 128, [3, 64, 1, 17] * 12 + [60]),
    (16, 16, 64, [2] * 70)])
def test_transposed_values_of_both_tiles(nh, nkv, hd, lens, splits):
    """Steps whose values are transposed 64 columns a block, from one partial sum and from several, and
    steps of many sequences that end inside a tile of 64 tokens, whose zeros begin at any column.  The
    sums are added in order in 32 bits and rounded once: what torch gives bit for bit."""
    from agave_b200 import kernels
    T, W = sum(lens), (nh + 2 * nkv) * hd
    part = rnd(splits, T, W, seed=4)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    pos = torch.cat([torch.arange(n) for n in lens]).int().to(DEV)
    seq = torch.cat([torch.full((n,), b) for b, n in enumerate(lens)]).int().to(DEV)
    cols = [(n + 63) // 64 * 64 for n in lens]
    vt = torch.full((nkv * hd, sum(cols) + 64), 7.0, dtype=torch.bfloat16, device=DEV)
    qkv = torch.empty(T, W, dtype=torch.bfloat16, device=DEV)
    kernels.qk_norm_rope_store(qkv, nh, nkv, hd, None, None, 1e-6, None, None, 0, pos, seq_index=seq,
                               partial=part, vt=vt, cu_seqlens=cu, max_len=max(lens))
    total = part[0].clone()
    for s in range(1, splits):
        total += part[s]
    assert torch.equal(qkv, total.to(torch.bfloat16))
    want = torch.zeros_like(vt)
    want[:, sum(cols):] = 7.0
    at = o = 0
    for n, c in zip(lens, cols):
        want[:, at:at + n] = qkv[o:o + n, (nh + nkv) * hd:].T
        at, o = at + c, o + n
    assert torch.equal(vt, want)


@pytest.mark.parametrize("dtype,T,N,K,splits,form", [
    (torch.float32, 1830, 2047, 4104, 1, (256, True)), (torch.float32, 5000, 4100, 1032, 1, (192, True)),
    (torch.float32, 300, 1150, 4104, 1, (128, True)), (torch.float32, 4100, 1001, 1160, 2, (256, False)),
    (torch.float32, 2051, 2301, 200, 1, (192, False)), (torch.float32, 400, 902, 2056, 2, (128, False)),
    (torch.float32, 700, 513, 4104, 2, (128, True)),
    (torch.bfloat16, 1030, 3001, 8200, 1, (256, True)), (torch.bfloat16, 700, 4100, 2056, 1, (192, True)),
    (torch.bfloat16, 200, 131, 72, 1, (128, True)), (torch.bfloat16, 3000, 1543, 200, 1, (256, False))])
def test_every_form_of_a_prompts_product(dtype, T, N, K, splits, form):
    """Each tile of a pair and of a CTA alone, by the plan's own choice: tokens, features and K that end
    inside a tile, rows whose stride is a multiple of four values and one that is not.  32-bit sums of
    bfloat16 products; into bfloat16 rounded once (2^-9)."""
    from agave_b200 import kernels
    assert kernels.linear_tc_prompt_form(T, N, K, splits, dtype) == form
    x = rnd(T, K, dtype=torch.bfloat16, seed=1)
    w = rnd(N, K, dtype=torch.bfloat16, seed=2, scale=K ** -0.5)
    ref = x.double() @ w.double().T
    for ld in (N,) if splits > 1 else (N + (-N) % 4, N + (-N) % 4 + 1):
        out = torch.full((splits, T, ld) if splits > 1 else (T + 1, ld), float("nan"), dtype=dtype, device=DEV)
        kernels.linear_tc(x, w, out if splits > 1 else out[:T, :N], splits=splits)
        assert kernels.linear_tc_status() == 0
        got = out.double().sum(0) if splits > 1 else out[:T, :N]
        assert rel_err(got, ref) < (1e-5 if dtype == torch.float32 else 4e-3)
        assert splits > 1 or (torch.isnan(out[T]).all() and torch.isnan(out[:, N:]).all())


@pytest.mark.parametrize("T,splits", [(600, 2), (3600, 1)])
def test_a_step_whose_products_are_cut_in_two(T, splits, tmp_path):
    """A prompt long enough for the rule of two ranges of K on the output and down products, and one
    beyond it: the norm behind them meets two partial sums or one.  Logits against the plain
    implementation in 32 bits; bfloat16 layers."""
    import os
    import sys
    sys.path.insert(0, os.path.dirname(os.path.abspath(__file__)))
    from plain import gemma3_plain as P
    from agave_b200 import kernels
    from agave_b200.engine.api import Engine
    from agave_b200.weights import write_model_folder
    cfg = {"architectures": ["Gemma3ForCausalLM"], "model_type": "gemma3_text", "num_hidden_layers": 2,
           "hidden_size": 512, "num_attention_heads": 8, "num_key_value_heads": 2, "head_dim": 256,
           "query_pre_attn_scalar": 256, "intermediate_size": 2304, "vocab_size": 384,
           "sliding_window": 100, "sliding_window_pattern": 2, "rope_local_base_freq": 10000.0,
           "rope_theta": 1000000.0, "rms_norm_eps": 1e-6, "max_position_embeddings": 4096,
           "eos_token_id": 1}
    for K in (2048, 2304):
        assert kernels.plan_splits(T, 512, K)[0] == splits
    write_model_folder(str(tmp_path), cfg, seed=3, dtype=torch.bfloat16)
    g = torch.Generator().manual_seed(4)
    tokens = torch.randint(2, 384, (T,), generator=g).tolist()
    pcfg, w = P.read_config(str(tmp_path)), P.read_weights(str(tmp_path))
    ref = P.forward_logits(pcfg, w, tokens)[-1].double()
    eng = Engine(str(tmp_path), dtype="bfloat16", max_tokens=4096)
    slot = eng.acquire()
    got = eng.step([(slot, tokens)], [[T - 1]]).reshape(384).double().cpu()
    assert kernels.linear_tc_status() == 0
    assert float((got - ref).norm() / ref.norm()) < 2e-2


@pytest.mark.parametrize("nh,nkv,hd,hdv", [(4, 1, 256, 256), (16, 16, 64, 64), (8, 2, 48, 80), (6, 6, 16, 16)])
@pytest.mark.parametrize("form", ["bias", "cap", "sinks", "blocks"])
def test_prompt_attention_of_many_short_sequences(nh, nkv, hd, hdv, form):
    """Sequences of a few tokens and of up to two half tiles of 64 keys in one step, with a bias by
    distance, a soft cap, a sink and blocks of positions, by either kernel.  Errors: P, the values and
    the result are bfloat16 (2^-9 each)."""
    from agave_b200 import kernels
    lens = [3, 1, 63, 7, 64, 2, 65, 31, 33, 127, 12, 5, 128, 4, 4, 4, 1, 1, 30]
    T, nan = sum(lens), float("nan")
    window = -40 if form == "blocks" else 0
    q, k = (rnd(T, n * hd, dtype=torch.bfloat16, seed=i, scale=0.5) for i, n in enumerate((nh, nkv)))
    v = rnd(T, nkv * hdv, dtype=torch.bfloat16, seed=3)
    cu = torch.tensor([0] + list(torch.tensor(lens).cumsum(0)), dtype=torch.int32, device=DEV)
    sinks = rnd(nh, seed=5) if form == "sinks" else None
    bias = rnd(nh, 50, seed=6) if form == "bias" else None
    cap = 2.0 if form == "cap" else 0.0
    for attend in (kernels.attention_prefill_tc, kernels.attention_prefill_mma):
        out = torch.full((T, nh * hdv), nan, dtype=torch.bfloat16, device=DEV)
        attend(q, k, v, out, cu, max(lens), nh, nkv, hd, 0.3, window, value_dim=hdv, sinks=sinks,
               dist_bias=bias, softcap=cap)
        assert kernels.attention_tc_status() == 0
        o = 0
        for n in lens:
            at = slice(o, o + n)
            qs = q[at].double().reshape(n, nh, hd).transpose(0, 1)
            ks = k[at].double().reshape(n, nkv, hd).transpose(0, 1).repeat_interleave(nh // nkv, 0)
            vs = v[at].double().reshape(n, nkv, hdv).transpose(0, 1).repeat_interleave(nh // nkv, 0)
            p = torch.arange(n, device=DEV)[:, None]
            j = torch.arange(n, device=DEV)[None, :]
            s = (qs @ ks.transpose(1, 2)) * 0.3
            if cap:
                s = cap * torch.tanh(s / cap)
            if bias is not None:
                s = s + bias.double()[:, (p - j).clamp(0, 49)]
            see = (j <= p) & (p // 40 == j // 40 if window else j >= 0)
            s = s.masked_fill(~see, float("-inf"))
            if sinks is not None:
                s = torch.cat([s, sinks.double()[:, None, None].expand(nh, n, 1)], -1)
            w = torch.softmax(s, -1)[..., :n]
            ref = (w @ vs).transpose(0, 1).reshape(n, nh * hdv)
            assert rel_err(out[at], ref) < 6e-3, n
            o += n


@pytest.mark.parametrize("lens", [[100], [300, 7], [12] * 12])
def test_a_score_scale_that_is_not_positive(lens, monkeypatch):
    """A negative scale with queries of the other sign is the same step: the tcgen05 attention, which
    takes positive scales alone, against the kernel that a negative one goes to, each launched by the
    C++ step function.  bfloat16 probabilities and results (2^-9) through two layers."""
    from dataclasses import replace
    from agave_b200 import Engine
    from agave_b200.config import resolve_architecture
    from agave_b200.models.decoder import decoder_param_specs
    from agave_b200.weights import random_tensors
    cfg = {"architectures": ["Gemma3ForCausalLM"], "model_type": "gemma3_text", "num_hidden_layers": 2,
           "hidden_size": 256, "num_attention_heads": 4, "num_key_value_heads": 2, "head_dim": 64,
           "query_pre_attn_scalar": 64, "intermediate_size": 512, "vocab_size": 384, "sliding_window": 100,
           "sliding_window_pattern": 2, "rope_local_base_freq": 10000.0, "rope_theta": 1000000.0,
           "rms_norm_eps": 1e-6, "max_position_embeddings": 1024, "eos_token_id": 1}
    made = resolve_architecture(cfg).config_class
    plain = made.to_model_spec
    tensors = random_tensors(decoder_param_specs(made.from_dict(cfg).to_model_spec()), 5, 0.05, 0.1,
                             torch.bfloat16, DEV)
    g = torch.Generator().manual_seed(6)
    prompts = [torch.randint(2, 384, (n,), generator=g).tolist() for n in lens]

    def logits(sign):
        t = {k: v.clone() for k, v in tensors.items()}
        if sign < 0:
            for k in t:
                if k.endswith("q_norm.weight"):
                    t[k] = -2 - t[k].float()           # (the norm's factor is 1 + w)

        def spec_of(self):
            spec = plain(self)
            return replace(spec, blocks=[replace(b, mixer=replace(b.mixer, scale=sign * b.mixer.scale))
                                         for b in spec.blocks])
        monkeypatch.setattr(made, "to_model_spec", spec_of)
        eng = Engine(None, _raw_config=cfg, _tensors=t, dtype="bfloat16", max_tokens=2048, max_batch=16)
        slots = [eng.acquire() for _ in prompts]
        return eng.step(list(zip(slots, prompts)), [list(range(n)) for n in lens]).double()

    a, b = logits(1), logits(-1)
    assert torch.isfinite(b).all()
    assert float((a - b).norm() / a.norm()) < 2e-2


@pytest.mark.parametrize("T,B,longest,nh,nkv,hd,fused,alone", [
    (1, 1, 1, 4, 1, 256, True, False), (100, 1, 100, 4, 1, 256, True, False), (100, 1, 100, 16, 16, 64, True, True),
    (300, 1, 300, 4, 1, 256, True, True), (192, 16, 12, 16, 16, 64, False, False),
    (1024, 16, 64, 32, 8, 64, False, False), (512, 16, 32, 32, 16, 128, True, False),
    (768, 64, 12, 16, 4, 128, True, True), (32, 8, 4, 16, 16, 64, False, False),
    (32, 8, 4, 4, 1, 256, True, False), (64, 1, 64, 16, 16, 16, True, True),
    (4096, 64, 64, 64, 8, 64, False, False)])
def test_which_kernel_attends_for_a_prompt(T, B, longest, nh, nkv, hd, fused, alone):
    """Either side of each line of the rule, with the values transposed by the q/k/v kernel and by one
    of their own."""
    from agave_b200 import kernels
    got = [bool(kernels.library().agv_attention_prefill_prefers_tc(T, B, longest, nh, nkv, hd, hd, vt))
           for vt in (1, 0)]
    assert got == [fused, alone]
