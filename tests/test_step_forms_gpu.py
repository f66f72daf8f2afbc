"""The kernels and forms of a step that a size or a pitch picks, at the sizes where they meet: clearing a new sequence's state, a grouped
product's search for its rows, the fused norm and router with several blocks a token, the norm that leaves three terms, rows gathered from a
pitch, the router's logits, the delta rule's preparation over runs of tokens, and queries, keys and values in one product."""
from __future__ import annotations

import pytest
import torch

import gpu_util as G

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def core():
    from moe_b200.ops import core

    core.lib()
    return core


@pytest.mark.parametrize("sizes", [[1], [7, 4096, 16384 // 4 + 1, 3], [5] * 33, [100_000, 0, 64]])
def test_clear_rows_clears_these_rows_and_nothing_else(core, sizes):
    bufs = [torch.ones(n + 2, device=DEV) for n in sizes]
    core.clear_rows([b[1:1 + n] for b, n in zip(bufs, sizes)])
    for b, n in zip(bufs, sizes):
        assert float(b.sum()) == 2.0 and float(b[0]) == 1.0 and float(b[-1]) == 1.0


def test_a_slot_used_again_starts_with_a_clear_state():
    from moe_b200.cache import KVCache, StateRequest

    cache = KVCache({}, {0: StateRequest((5,)), 1: StateRequest((3, 9), torch.bfloat16), 2: StateRequest((1,), torch.int32)}, 64, 2,
                    torch.bfloat16, DEV)
    a = cache.acquire()
    for i in range(3):
        cache.state(i).fill_(1)
    cache.release(a)
    b = cache.acquire()
    for i in range(3):
        t = cache.state(i).float()
        assert float(t[b].abs().sum()) == 0.0 and int((t == 1).sum()) == t.numel() - t[b].numel()


@pytest.mark.parametrize("T,H", [(1, 4), (300, 2048), (257, 264), (3, 12032)])
@pytest.mark.parametrize("with_delta", [True, False])
def test_the_norm_that_leaves_three_terms(core, T, H, with_delta):
    """The same as norm and split, to the bit; a row pitch that is no whole unit is left to them."""
    torch.manual_seed(T)
    x, w = torch.randn(T, H, device=DEV), torch.randn(H, device=DEV)
    delta = torch.randn(T, H, device=DEV) if with_delta else None
    x1, x2, o32, st = x.clone(), x.clone(), torch.empty(T, H, device=DEV), core.new_status(DEV)
    core.rmsnorm(x1, w, 1e-6, delta=delta, out32=o32, status=st)
    got = core.rmsnorm_split(x2, w, 1e-6, delta=delta, status=st)
    assert torch.equal(x1, x2)
    if T >= 256:        # (fewer rows: the norm beside it is another instance, whose products may be contracted otherwise)
        assert torch.equal(got, core.split3(o32))
    y = got.float().view(T, 3, H)
    assert torch.allclose((y[:, 0] + y[:, 1]) + y[:, 2], o32, rtol=3e-7, atol=1e-12) and int(st[0]) == 0
    assert core.rmsnorm_split(torch.randn(2, 6, device=DEV), torch.ones(6, device=DEV), 1e-6, status=st) is None


def test_gather_rows_from_a_pitch(core):
    from moe_b200.ops import tc

    src, st = torch.randn(9, 3 * 72, device=DEV).bfloat16(), core.new_status(DEV)
    rows = torch.tensor([8, 0, 3, 3], dtype=torch.int32, device=DEV)
    for lo in (0, 72):
        assert torch.equal(tc.gather_rows(src[:, lo:lo + 72], rows, 4, st), src[:, lo:lo + 72][rows.long()])
    assert int(st[0]) == 0


@pytest.mark.parametrize("groups", [1, 31, 33, 70, 300])
def test_a_grouped_product_finds_its_rows_among_any_number_of_groups(groups):
    """Few rows a group, empty groups among them, tiles that end inside a group; in one CTA a tile and on persistent CTAs."""
    from moe_b200.ops import core as c, tc

    torch.manual_seed(groups)
    counts = [0 if g % 5 == 2 else 1 + (g * 7) % 23 for g in range(groups)]
    offs = torch.tensor([0] + torch.tensor(counts).cumsum(0).tolist(), dtype=torch.int32, device=DEV)
    M, K, N = sum(counts), 136, 72
    x, w, st = torch.randn(M, K, device=DEV).bfloat16(), torch.randn(groups, N, K, device=DEV).bfloat16(), c.new_status(DEV)
    ref = torch.cat([x[int(offs[g]):int(offs[g + 1])].double() @ w[g].double().T for g in range(groups)])
    for bn in (16, 32, 128):
        for early in (False, True):
            out = torch.full((M, N), float("nan"), device=DEV)
            assert tc.gemm_tc(x, w, out, group_offsets=offs, bn=bn, splits=1, status=st, early_offsets=early)
            # 136 products of bfloat16 numbers of size 1, added in 32 bits
            assert float((out.double() - ref).abs().max()) < 136 * 8 * 2.0 ** -23 * 8, (bn, early)
    assert int(st[0]) == 0


@pytest.mark.parametrize("S", [2, 3, 4, 5, 6, 7, 8])
@pytest.mark.parametrize("swiglu", [False, True])
@pytest.mark.parametrize("grouped", [False, True])
def test_k_splits_of_few_rows_push_or_are_read(core, S, swiglu, grouped):
    """Every number of rows on both sides of the rule and of the receive buffer's size, groups that fill a tile and empty ones: against 64 bits, a row
    the same to the bit in either form, nothing written past the last row."""
    from moe_b200.ops import tc

    torch.manual_seed(S)
    groups, K, N, st = 4 if grouped else 1, 128 * S - 8, 136, core.new_status(DEV)       # two blocks of k a split, the last one ragged
    shape = (groups, (2 if swiglu else 1) * N, K) if grouped else ((2 if swiglu else 1) * N, K)
    rows, w = torch.randn(24, K, device=DEV).bfloat16(), (torch.randn(shape, device=DEV) * K ** -0.5).bfloat16()
    wide = w.view(groups, -1, K)

    def run(x, counts):
        M, out = x.shape[0], torch.full((x.shape[0] + 3, N), 7.0, device=DEV)
        offs = torch.tensor([0] + torch.tensor(counts).cumsum(0).tolist(), dtype=torch.int32, device=DEV) if grouped else None
        assert tc.gemm_tc(x, w, out, swiglu=swiglu, group_offsets=offs, bn=16, splits=S, status=st)
        assert bool((out[M:] == 7.0).all())
        return out[:M]

    for M in range(1, 18):
        x = rows[:M].contiguous()
        # one group of M rows among empty ones (a grouped product of more than 16 rows in all has another form)
        counts = [0, M, 0, 0]
        got = run(x, counts)
        ref = x.double() @ wide[1 if grouped else 0].double().T
        slack = (K + S) * 2.0 ** -24 * (x.double().abs() @ wide[1 if grouped else 0].double().abs().T)      # exact products, K + S sums in 32 bits
        if swiglu:
            a, b, ea, eb = ref[:, :N], ref[:, N:], slack[:, :N], slack[:, N:]
            ref = torch.nn.functional.silu(a) * b
            slack = 1.1 * ea * b.abs() + a.abs() * eb + ea * eb + 1e-6 * ref.abs()       # |silu'| <= 1.1, |silu(a)| <= |a|
        assert bool(((got.double() - ref).abs() <= slack).all()), M
        more = run(torch.cat([x, rows[M:]]) if grouped else rows[:16 if M <= 16 else 24].contiguous(), [0, M, 0, 24 - M])
        assert torch.equal(more[:M], got), M
    assert int(st[0]) == 0


@pytest.mark.parametrize("T", [1, 2, 3, 4, 5, 7, 8])
@pytest.mark.parametrize("E,k,H,post", [(61, 4, 2048, False), (16, 2, 2056, True), (256, 8, 4104, False), (3, 3, 40, True)])
def test_norm_and_router_with_several_blocks_a_token(core, T, E, k, H, post):
    """Against 64 bits, for every number of blocks a token (eight blocks among the tokens)."""
    torch.manual_seed(T + E)
    x0, a, b = (torch.randn(T, H, device=DEV) for _ in range(3))
    w, wr = 1 + 0.1 * torch.randn(H, device=DEV), (torch.randn(E, H, device=DEV) * H ** -0.5).bfloat16()
    wsg = None if post else (torch.randn(H, device=DEV) * H ** -0.5).bfloat16()
    seq, st, x = torch.zeros(T, dtype=torch.int32, device=DEV), core.new_status(DEV), x0.clone()
    if T > 2:
        seq[1] = -1
    if post:
        res = core.norm_route(x, a, None, 0.0, wr, k, True, 1.0, bf16=True, seq_of_token=seq, status=st, delta_b=b, sa=0.5, sb=0.25,
                              post=(w, 1e-5), weight_input=True)
        y = 0.5 * a.double() + 0.25 * b.double()
        ref = x0.double() + y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5) * w.double()
        assert torch.allclose(x.double(), ref, rtol=1e-5, atol=1e-6)
        row = x
    else:
        res = core.norm_route(x, a, w, 1e-5, wr, k, True, 1.0, bf16=True, shared_gate_w=wsg, seq_of_token=seq, status=st)
        assert torch.equal(x, x0 + a)
        y = x.double()
        row = (y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5) * w.double()).float()
        assert float((res[1].float() - row).abs().max()) <= 2.0 ** -8 * float(row.abs().max())
    out32, out16, idx, wt, sg, offs, sorted_token, pos, xs = res
    live = (seq >= 0).tolist()
    probs = torch.softmax(row.double() @ wr.double().T, -1)
    pairs, want = idx.tolist(), torch.topk(probs, k, -1)
    flat = [(e, t * k + j) for t in range(T) for j, e in enumerate(pairs[t]) if live[t]]
    for t in range(T):
        if not live[t]:
            assert pairs[t] == [-1] * k and float(wt[t].abs().sum()) == 0.0
            continue
        # (a pick of another expert only where the two are as likely to rounding)
        assert torch.allclose(probs[t][idx[t].long()], want.values[t], rtol=1e-5)
        ref_w = probs[t][idx[t].long()] / probs[t][idx[t].long()].sum()
        assert torch.allclose(wt[t].double(), ref_w, rtol=1e-5)
        if sg is not None:
            assert abs(float(sg[t]) - float(torch.sigmoid(row[t].double() @ wsg.double()))) < 1e-5
    order = {p: i for i, (_, p) in enumerate(sorted(flat))}              # places: by expert, then in pair order
    assert pos.reshape(-1).tolist() == [order.get(p, -1) for p in range(T * k)]
    assert offs.tolist() == [sum(e < g for e, _ in flat) for g in range(E + 1)]
    for p, i in order.items():
        assert int(sorted_token[i]) == p // k
        src = row[p // k] * (wt.reshape(-1)[p] if post else 1.0)
        assert float((xs[i].float() - src).abs().max()) <= 2.0 ** -8 * float(src.abs().max())
    assert int(st[0]) == 0


@pytest.mark.parametrize("d,dv,taps,channel", [(128, 128, 4, True), (64, 40, 2, False), (36, 128, 3, True), (100, 12, 4, False)])
def test_the_delta_rules_preparation_over_runs_of_tokens(core, d, dv, taps, channel):
    """A step of 128 rows and more goes over runs of eight tokens, which sequences begin and end inside of; a step's pieces of fewer rows
    do not: the same to the bit, rows of no sequence among them."""
    torch.manual_seed(d)
    H, Gk, lens = 3, 3, [1, 61, 2, 75, 20]
    ch, T = 2 * Gk * d + H * dv, sum(lens)
    ld = ch + 2 * H + (-(ch + 2 * H)) % 4
    proj, tw = torch.randn(T, ld, device=DEV), torch.randn(taps, ch, device=DEV)
    a_log, bias = torch.randn(H, device=DEV), torch.randn(H * d if channel else H, device=DEV)
    a_rows = torch.randn(T, H * d, device=DEV) if channel else None
    start = torch.randn(len(lens) + 1, ((taps - 1) * ch + 3) // 4 * 4, device=DEV)
    kw = dict(heads=H, kv_heads=Gk, d=d, dv=dv, b_at=ch, a_at=ch + H, eps=1e-6, q_scale=d ** -0.5)

    def run(proj, a_rows, batch):
        n = proj.shape[0]
        out, step = torch.full((n, ch), float("nan"), device=DEV), torch.full((n, 2 * H), float("nan"), device=DEV)
        decay = torch.full((n, H * d), float("nan"), device=DEV) if channel else None
        core.delta_prepare(proj, tw, a_log, bias, start.clone(), batch, out, step, a_rows=a_rows, decay=decay, **kw)
        return [t for t in (out, step, decay) if t is not None]

    whole = G.make_batch(DEV, list(range(len(lens))), [0] * len(lens), lens)
    got = run(proj, a_rows, whole)
    at = 0
    for i, n in enumerate(lens):
        alone = run(proj[at:at + n].contiguous(), a_rows[at:at + n].contiguous() if channel else None, G.make_batch(DEV, [i], [0], [n]))
        for g, w in zip(got, alone):
            assert torch.equal(g[at:at + n], w), i
        at += n
    whole.seq_of_token[140:] = -1                        # rows of no sequence: finite, and the others as before
    for g, w in zip(run(proj, a_rows, whole), got):
        assert torch.equal(g[:140], w[:140]) and bool(g[140:].isfinite().all())


@pytest.mark.parametrize("T", [9, 64, 65, 131, 256])
@pytest.mark.parametrize("E,H", [(60, 2048), (17, 264), (33, 3592), (4, 8)])
@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
def test_router_logits_of_nine_tokens_and_more(core, T, E, H, wdt):
    """Picks and weights against 64 bits; tokens and router rows that fill no whole block."""
    torch.manual_seed(T + E)
    h, wr = torch.randn(T, H, device=DEV), (torch.randn(E, H, device=DEV) * H ** -0.5).to(wdt)
    wsg, k = (torch.randn(H, device=DEV) * H ** -0.5).to(wdt), min(3, E)
    idx, w, sg = torch.empty(T, k, dtype=torch.int32, device=DEV), torch.empty(T, k, device=DEV), torch.empty(T, device=DEV)
    core.router(h, wr, k, False, 1.0, idx, w, shared_gate_w=wsg, shared_gate=sg)
    probs = torch.softmax(h.double() @ wr.double().T, -1)
    # logits of size 1, H products added in 32 bits by 32 lanes: off by some 1e-6
    assert torch.allclose(probs.gather(1, idx.long()), torch.topk(probs, k, -1).values, rtol=2e-5)
    assert torch.allclose(w.double(), probs.gather(1, idx.long()), rtol=2e-5)
    assert torch.allclose(sg.double(), torch.sigmoid(h.double() @ wsg.double()), rtol=2e-5)


@pytest.mark.parametrize("T,E", [(65, 17), (256, 128), (131, 1), (301, 33)])
@pytest.mark.parametrize("H", [12280, 12288, 12296, 24576, 24840])
@pytest.mark.parametrize("wdt", [torch.float32, torch.bfloat16])
def test_router_logits_of_rows_wider_than_shared_memory(core, T, E, H, wdt):
    """One slab of 12,288 features and several, the last one of one unit; without scratch, which 257 tokens and more otherwise use."""
    torch.manual_seed(T + H)
    h, wr, wsg = torch.randn(T, H, device=DEV), (torch.randn(E, H, device=DEV) * H ** -0.5).to(wdt), torch.randn(H, device=DEV).to(wdt)
    out = torch.full((T, E + 1), float("nan"), device=DEV)
    core._ok(core.lib().moe_router_logits(core._p(h), core._p(wr), core._p(wsg), core._dt(wr), T, H, E, core._p(out), None, 0,
                                          core._stream()), "router_logits")
    rows = torch.cat([wr, wsg[None]]).double().T
    # a lane adds H / 32 products, the lanes' sums meet in five steps: each rounds by half a unit of at most all terms' size
    bound = (H / 32 + 5) * 2.0 ** -24 * (h.double().abs() @ rows.abs())
    assert bool(((out.double() - h.double() @ rows).abs() <= bound).all())


@pytest.mark.parametrize("M,nh,nkv,K,bias,window", [(257, 4, 4, 264, True, None), (300, 7, 1, 512, False, None), (513, 3, 2, 136, True, 128),
                                                    (3100, 2, 1, 520, True, None), (3073, 3, 3, 256, False, 256)])
def test_queries_keys_and_values_in_one_product(core, M, nh, nkv, K, bias, window):
    """The same as the product, then rotation, split and append, to the bit: single CTAs and pairs, an odd number of heads, a ring, rows of
    no sequence, sequences that go on."""
    from moe_b200.cache import KVCache, KVRequest
    from moe_b200.ops import tc

    torch.manual_seed(M)
    x, w = torch.randn(M, K, device=DEV).bfloat16(), (torch.randn((nh + 2 * nkv) * 128, K, device=DEV) * K ** -0.5).bfloat16()
    b = torch.randn((nh + 2 * nkv) * 128, device=DEV) if bias else None
    freq = 10000.0 ** (-torch.arange(64, device=DEV, dtype=torch.float32) / 64)
    lens, starts, st = [100, M - 107, 7], [0, 5, 77], core.new_status(DEV)
    batch = G.make_batch(DEV, [1, 0, 2], starts, lens)
    batch.seq_of_token[100 + 40] = -1
    caches = []
    for fused in (False, True):
        cache = KVCache({0: KVRequest(nkv, 128, window)}, {0: None}, M + 1024, 3, torch.bfloat16, DEV)
        for _ in range(3):
            cache.acquire()
        for slot, n0, n in zip([1, 0, 2], starts, lens):
            G.give_pages(cache, slot, n0 + n)
        cache.groups[0].storage.fill_(3.0)
        view = cache.view(0)
        q, k, v = (torch.full((M, n, 128), 9.0, device=DEV, dtype=torch.bfloat16) for n in (nh, nkv, nkv))
        if fused:
            angles, rows = core.rope_angles(batch, freq, 64, view, st)
            assert tc.gemm_qkv(x, w, b, angles, rows, q, k, v, view, nh=nh, nkv=nkv, status=st)
        else:
            out = torch.empty(M, w.shape[0], device=DEV)
            assert tc.gemm_tc(x, w, out, bias=b, bn=256, splits=1, status=st)
            core.rope_split(out, batch.pos, freq, nh, nkv, 128, 128, q, k, v, commit=None)
        caches.append((q, k, v, rows if fused else None))
    for got, want in zip(caches[1][:3], caches[0][:3]):
        assert torch.equal(got, want)
    # the appended rows, each where the page table says
    grp, rows = cache.groups[0], caches[1][3].tolist()
    kc, vc = (t.reshape(-1, 128) for t in (view.k, view.v))
    at, written = 0, {}
    for i, (slot, s0, n) in enumerate(zip([1, 0, 2], starts, lens)):
        for j in range(n):
            t, pos = at + j, s0 + j
            held = t != 140 and (grp.ring == 0 or pos >= s0 + n - grp.ring)
            place = pos % grp.ring if grp.ring else pos
            want = int(grp.table[slot, place // 64]) * nkv * 64 + place % 64 if held else -1
            if t % 13 == 0 or n < 20:
                assert rows[t] == want, (t, pos)
            if rows[t] >= 0:
                written[rows[t]] = t
        at += n
    for r, t in list(written.items())[::11]:
        for h in range(nkv):
            assert torch.equal(kc[r + h * 64], caches[1][1][t, h]) and torch.equal(vc[r + h * 64], caches[1][2][t, h])
    untouched = kc.shape[0] - nkv * len(written)
    assert int((kc == 3.0).all(-1).sum()) >= untouched and int(st[0]) == 0


def test_long_steps_project_rotate_and_append_in_one_product_as_one_by_one(monkeypatch):
    """A model whose layers share angles and cache rows within a step (windowed layers with a ring of their own among full ones): a prompt of 1,280
    rows and more, a continued step of two sequences, another prompt, then a step of decoding, with the product that rotates and appends
    and without it.  Logits and the whole cache to the bit."""
    import moe_b200
    from moe_b200.ops import tc

    cfg = dict(architectures=["Qwen2MoeForCausalLM"], model_type="qwen2_moe", num_hidden_layers=4, hidden_size=264, num_attention_heads=3,
               num_key_value_heads=1, head_dim=128, num_experts=4, num_experts_per_tok=2, norm_topk_prob=False, decoder_sparse_step=1,
               moe_intermediate_size=72, shared_expert_intermediate_size=136, intermediate_size=136, vocab_size=301, rope_theta=1e4,
               rms_norm_eps=1e-6, use_sliding_window=True, sliding_window=200, max_window_layers=2, tie_word_embeddings=False)
    model = moe_b200.random_model(cfg, seed=3, dtype="bfloat16", device=DEV)
    ids = torch.randint(0, 301, (6000,), generator=torch.Generator().manual_seed(1)).tolist()
    fused, taken = tc.gemm_qkv, []

    def counted(*args, **kw):
        taken.append((args[0].shape[0], args[4] is not None))         # rows, and whether keys and values go to the cache at once
        return fused(*args, **kw)

    def steps():
        engine = moe_b200.Engine(model, max_tokens=8192, max_slots=2)
        a, b = engine.new_sequence(), engine.new_sequence()
        out = [engine.step(s, t).clone() for s, t in (([a], [ids[:1300]]), ([a, b], [ids[1300:2700], ids[2700:2750]]),
                                                      ([b], [ids[3000:4281]]), ([a, b], [[7], [9]]))]
        engine.rt.check()
        return out, [g.storage.clone() for g in engine.cache.groups], [g.ring for g in engine.cache.groups]

    monkeypatch.setattr(tc, "gemm_qkv", counted)
    got, kept, rings = steps()
    assert len(rings) == 2 and sum(r > 0 for r in rings) == 1
    # four layers each: a prompt appends everywhere at once, a step that goes on does so but in the ring of the two windowed layers
    assert sorted(taken) == sorted([(1300, True)] * 4 + [(1450, True), (1450, False), (1281, True), (1281, False)] * 2)
    monkeypatch.setattr(tc, "takes_qkv", lambda x, w: False)
    del taken[:]
    want, held, _ = steps()
    assert not taken
    for g, w in zip(got + kept, want + held):
        assert torch.equal(g, w)


@pytest.mark.parametrize("dt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nh,nkv,hd,rot", [(3, 1, 128, 128), (5, 5, 24, 16)])
def test_rope_split_zeroes_the_rows_of_no_sequence_and_no_others(core, dt, nh, nkv, hd, rot):
    from moe_b200.cache import KVCache, KVRequest

    T, st = 90, core.new_status(DEV)
    cache = KVCache({0: KVRequest(nkv, hd, None)}, {0: None}, 256, 2, dt, DEV)
    cache.acquire()
    G.give_pages(cache, 0, T)
    batch = G.make_batch(DEV, [0], [0], [T])
    none = [0, 17, 88, 89]
    batch.seq_of_token[none] = -1
    qkv, freq = torch.randn(T, (nh + 2 * nkv) * hd, device=DEV), torch.rand(rot // 2, device=DEV)
    q, k, v = (torch.empty(T, n, hd, device=DEV, dtype=dt) for n in (nh, nkv, nkv))
    ctx = torch.full((T, nh * hd), float("nan"), device=DEV, dtype=dt)
    assert core.rope_split(qkv, batch.pos, freq, nh, nkv, hd, rot, q, k, v, commit=(cache.view(0), batch), status=st, zero=ctx)
    assert torch.equal(ctx[none], torch.zeros_like(ctx[none])) and int(ctx.isnan().all(1).sum()) == T - len(none) and int(st[0]) == 0


@pytest.mark.parametrize("E,k", [(4, 3), (70, 8), (33, 1), (5, 5)])
@pytest.mark.parametrize("score", ["softmax", "sigmoid"])
@pytest.mark.parametrize("norm", [False, True])
def test_picks_from_logits_that_are_infinite_or_no_numbers(core, E, k, score, norm):
    """The best score first, the lowest expert among equals, a score that is no number never; where none is left, expert j mod E with weight 0."""
    inf, nan = float("inf"), float("nan")
    rows = [[0.0] * E, [nan] * E, [-inf] * E, [inf] * E, [nan] + [-1.0] * (E - 1), [-inf] * (E - 1) + [2.0], [inf] + [0.5] * (E - 1),
            [nan, inf] + [-inf] * (E - 2), [nan] * (E - 2) + [3.0, 3.0], [-200.0] * (E - 1) + [-0.0], [1e38, -1e38] + [0.0] * (E - 2)]
    logits = torch.tensor(rows)
    idx, w = torch.empty(len(rows), k, dtype=torch.int32, device=DEV), torch.empty(len(rows), k, device=DEV)
    core.router_topk(logits.to(DEV), k, norm, 1.0, idx, w, num_experts=E, score=score)
    for i, lg in enumerate(logits):
        # (scores that vanish in 32 bits are equal)
        sc = (torch.softmax(lg.double(), 0) if score == "softmax" else 1 / (1 + torch.exp(-lg).double())).float().tolist()
        left, picks, weights = set(range(E)), [], []
        for j in range(k):
            best = max((e for e in left if sc[e] == sc[e]), key=lambda e: (sc[e], -e), default=None)
            picks.append(j % E if best is None else best)
            weights.append(0.0 if best is None else sc[best])
            left.discard(picks[-1])
        total = max(sum(weights), 1e-20) if norm else 1.0
        assert idx[i].tolist() == picks, i
        # E exponentials and their sum, in 32 bits
        assert torch.allclose(w[i].double().cpu(), torch.tensor([x / total for x in weights], dtype=torch.float64), rtol=2e-5, atol=1e-30), i
