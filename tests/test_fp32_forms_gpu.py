"""The forms of the 32-bit kernels that a size picks, at the sizes where they meet: products of few and of many rows
(16-byte operands; the tile heights; group counts), attention of 128 queries a block, the delta rule over chunks of
sixteen tokens and the mLSTM memory over chunks of sixty-four beside their forms of four, against float64."""
import math

import numpy as np
import pytest
import torch

import gpu_util as G

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 2.0 ** -24


@pytest.fixture(scope="module")
def core():
    from moe_b200.ops import core

    core.lib()
    return core


def bound(a, w):
    """An output's products are added 256 at a time, then the chunks' sums: every addition and product is off by at most
    half a unit, so |error| <= (256 + chunks + 1) 2^-24 sum |a w| (first order)."""
    K = a.shape[-1]
    return (min(K, 256) + -(-K // 256) + 2) * EPS * (a.double().abs() @ w.double().abs().T) + 1e-30


@pytest.mark.parametrize("K,N", [(4, 1), (252, 130), (256, 16), (260, 31), (1408, 129), (2052, 17), (5632, 48)])
def test_a_row_is_the_same_to_the_bit_for_every_number_of_rows(core, K, N):
    torch.manual_seed(K + N)
    a, w, b = torch.randn(330, K, device=DEV), torch.randn(N, K, device=DEV), torch.randn(N, device=DEV)
    st = core.new_status(DEV)
    many = torch.empty(330, N, device=DEV)
    core.gemm_generic(a, w, many, bias=b, status=st)
    assert bool(((many.double() - (a.double() @ w.double().T + b.double())).abs() <= bound(a, w) + 2 * EPS * many.double().abs()).all())
    for M in (1, 7, 8, 9, 16, 17, 40, 41, 64, 65, 160, 161):
        out = torch.full((M + 1, N), float("nan"), device=DEV)
        core.gemm_generic(a[:M], w, out[:M], bias=b, status=st)
        assert torch.equal(out[:M], many[:M]), M
        assert bool(out[M].isnan().all())
    # rows that do not start on 16 bytes take the plain kernels, in the same order of summation
    off = torch.empty(330 * K + 1, device=DEV)[1:].view(330, K)
    off.copy_(a)
    for M in (3, 330):
        out = torch.empty(M, N, device=DEV)
        core.gemm_generic(off[:M], w, out, bias=b, status=st)
        assert torch.equal(out, many[:M]), M
    assert int(st[0]) == 0


@pytest.mark.parametrize("counts", [[3, 0, 1, 8, 9, 0, 17], [0] * 40 + [5, 0, 33], [70, 0, 3, 129, 1], [300, 5], [0, 0, 64]])
def test_grouped_rows_gathered(core, counts):
    torch.manual_seed(sum(counts))
    E, N, K, S = len(counts), 140, 516, 50
    a, w = torch.randn(S, K, device=DEV), torch.randn(E, N, K, device=DEV)
    offs = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32, device=DEV)
    M = sum(counts)
    rows = torch.randint(0, S, (M,), device=DEV, dtype=torch.int32)
    st = core.new_status(DEV)
    out = torch.full((M, N), float("nan"), device=DEV)
    core.gemm_generic(a, w, out, a_rows=rows, group_offsets=offs, status=st)
    at = 0
    for g, c in enumerate(counts):
        x = a[rows[at:at + c].long()]
        assert bool(((out[at:at + c].double() - x.double() @ w[g].double().T).abs() <= bound(x, w[g])).all()), g
        at += c
    assert int(st[0]) == 0


@pytest.mark.parametrize("hd,nh,nkv", [(128, 2, 1), (64, 3, 3)])
@pytest.mark.parametrize("before,new", [([0, 0], [128, 129]), ([5, 300], [257, 130]), ([64], [511]), ([1000, 0, 127], [150, 260, 128])])
@pytest.mark.parametrize("opt", [{}, {"window": 100}, {"window": 130, "keep": 70}, {"chunk": 96, "softcap": 5.0}, {"sink": True},
                                 {"sigmoid": True}, {"sigmoid": True, "chunk": 96}])
def test_attention_of_many_new_tokens(core, hd, nh, nkv, before, new, opt):
    from moe_b200.cache import KVCache, KVRequest

    torch.manual_seed(hd + sum(new))
    window, keep, chunk, cap = opt.get("window"), opt.get("keep", 0), opt.get("chunk", 0), opt.get("softcap", 0.0)
    B = len(new)
    ring = window or chunk or None
    cache = KVCache({0: KVRequest(nkv, hd, ring, keep=keep) if keep else KVRequest(nkv, hd, ring)}, {0: None}, max_tokens=64 * 60,
                    max_slots=B + 1, dtype=torch.float32, device=DEV)
    cache.groups[0].storage.fill_(3e30)
    view, slots, st = cache.view(0), [cache.acquire() for _ in range(B)], core.new_status(DEV)
    K, V = ([torch.randn(a + b, nkv, hd, device=DEV) for a, b in zip(before, new)] for _ in range(2))
    Q = [2 * torch.randn(b, nh, hd, device=DEV) for b in new]
    live = [i for i in range(B) if before[i]]
    for i in live:
        G.give_pages(cache, slots[i], before[i])
    if live:
        b0 = G.make_batch(DEV, [slots[i] for i in live], [0] * len(live), [before[i] for i in live])
        core.kv_commit(*(torch.cat([x[i][:before[i]] for i in live]).contiguous() for x in (K, V)), view, b0, st)
    for i in range(B):
        G.give_pages(cache, slots[i], before[i] + new[i])
    batch = G.make_batch(DEV, slots, before, new)
    q, kn, vn = torch.cat(Q).contiguous(), *(torch.cat([x[i][before[i]:] for i in range(B)]).contiguous() for x in (K, V))
    out, bias = torch.full((q.shape[0], nh * hd), float("nan"), device=DEV), torch.randn(nh, device=DEV)
    sink = core.SigmoidWeights(bias) if opt.get("sigmoid") else opt.get("sink", False)
    assert core.attention_tiled(q, kn, vn, view, batch, out, nh=nh, window=window, scale=hd ** -0.5, use_local=True, status=st,
                                chunk=chunk, softcap=cap, sink=sink, keep=keep)
    at = 0
    for i in range(B):
        n, T = new[i], before[i] + new[i]
        p, j = torch.arange(before[i], T, device=DEV)[:, None], torch.arange(T, device=DEV)[None]
        seen = j <= p
        if chunk:
            seen &= j >= p // chunk * chunk
        elif window:
            seen &= (j > p - window) | (j < keep)
        for h in range(nh):
            s = Q[i][:, h].double() @ K[i][:, h // (nh // nkv)].double().T * hd ** -0.5
            s = cap * torch.tanh(s / cap) if cap else s
            s = s.masked_fill(~seen, -math.inf)
            if opt.get("sink"):
                s = torch.cat([s, torch.zeros(n, 1, dtype=s.dtype, device=DEV)], 1)
            weights = torch.sigmoid(s + bias[h].double()) if opt.get("sigmoid") else torch.softmax(s, -1)[:, :T]
            values = V[i][:, h // (nh // nkv)].double()
            ref, size = weights @ values, (weights @ values.abs()).clamp(min=1.0) if opt.get("sigmoid") else 1.0
            got = out[at:at + n, h * hd:(h + 1) * hd].double()
            # scores of up to about 30 are off by 128 half units at most, so a weight is by 30 * 128 * 2^-24 of itself (sigmoid
            # weights do not sum to 1: an output is off by that part of its terms)
            assert float(((got - ref).abs() / size).max()) < 3e-4, (i, h)
        at += n
    assert int(st[0]) == 0


@pytest.mark.parametrize("channel", [True, False])
@pytest.mark.parametrize("H,Gk,d,dv,lens", [(2, 1, 128, 128, [16, 1, 33]), (3, 3, 64, 96, [15, 17, 200]), (2, 2, 12, 20, [31, 48, 5]),
                                            (2, 1, 100, 36, [64, 3]), (1, 1, 128, 8, [130])])
def test_the_delta_rule_over_chunks_and_four_at_a_time(core, channel, H, Gk, d, dv, lens):
    g = torch.Generator(device=DEV).manual_seed(d + dv)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    T, B = sum(lens), len(lens)
    unit = torch.nn.functional.normalize
    q, k, v = unit(r(T, Gk, d), dim=-1) * d ** -0.5, unit(r(T, Gk, d), dim=-1), r(T, H, dv)
    beta, lg = torch.sigmoid(2 * r(T, H)), -torch.nn.functional.softplus(3 * r(T, H))
    decay = torch.exp(-torch.nn.functional.softplus(3 * r(T, H * d)))
    decay[::5, ::3] = 0.0                                   # a channel that forgets everything, and one that forgets nothing
    decay[1::5, 1::3] = 1.0
    qkv = torch.cat([x.reshape(T, -1) for x in (q, k, v)], 1).contiguous()
    step = torch.cat([beta, torch.zeros_like(lg) if channel else lg], 1).contiguous()
    batch = G.make_batch(DEV, list(range(1, B + 1)), [0] * B, lens)
    start = r(B + 2, 3 + H * d * dv + 1)[:, :4 + H * d * dv].contiguous()
    owner = torch.arange(H, device=DEV) // (H // Gk)
    for chunks in (False, True):
        state, o = start.clone(), torch.full((T, H * dv), float("nan"), device=DEV)
        core.delta_scan(qkv, step, state, batch, o, heads=H, kv_heads=Gk, d=d, dv=dv, offset=4, decay=decay if channel else None,
                        chunks=chunks)
        assert torch.equal(state[0], start[0]) and torch.equal(state[B + 1], start[B + 1]) and torch.equal(state[:, :4], start[:, :4])
        at = 0
        for i, n in enumerate(lens):
            S, ref = start[i + 1, 4:].double().view(H, d, dv), []
            for t in range(at, at + n):
                S = S * (decay[t].double().view(H, d, 1) if channel else torch.exp(lg[t].double())[:, None, None])
                kk, qq = k[t, owner].double(), q[t, owner].double()
                S = S + kk[:, :, None] * (beta[t].double()[:, None] * (v[t].double() - torch.einsum("hdv,hd->hv", S, kk)))[:, None]
                ref.append(torch.einsum("hdv,hd->hv", S, qq))
            ref = torch.stack(ref)
            got = o[at:at + n].view(n, H, dv).double()
            # a state of norm about 10 whose every element passes some d + 16 roundings a chunk
            assert float((got - ref).abs().max()) < 3e-5 * float(ref.abs().max()), (chunks, i)
            assert float((state[i + 1, 4:].double().view(H, d, dv) - S).abs().max()) < 3e-5 * float(S.abs().max()), (chunks, i)
            at += n


@pytest.mark.parametrize("H,d,dv,lens", [(2, 64, 128, [1, 63, 64]), (3, 12, 20, [65, 130]), (1, 100, 36, [200]), (2, 128, 260, [70, 5])])
def test_the_memory_over_chunks_and_four_at_a_time(core, H, d, dv, lens):
    g = torch.Generator(device=DEV).manual_seed(d + dv)
    T, B, cap = sum(lens), len(lens), 9.0
    at = {"q": 0, "k": H * d, "v": 2 * H * d, "i": 2 * H * d + H * dv, "f": 2 * H * d + H * dv + H}
    proj = torch.randn(T, -(-(at["f"] + H) // 4) * 4, device=DEV, generator=g)
    ib, fb = (torch.randn(H, device=DEV, generator=g) + b for b in (-0.5, 2.0))
    floats = core.mlstm_state_floats(H, d, dv)
    copies = -(-dv // 16)
    start = torch.zeros(B + 2, -(-(floats + 4) // 4) * 4, device=DEV)
    start[:, 4:4 + H * d * dv] = 0.3 * torch.randn(B + 2, H * d * dv, device=DEV, generator=g)
    norm = 0.3 * torch.randn(B + 2, 1, H * d, device=DEV, generator=g)
    start[:, 4 + H * d * dv:4 + H * d * (dv + copies)] = norm.expand(-1, copies, -1).reshape(B + 2, -1)
    batch = G.make_batch(DEV, list(range(1, B + 1)), [0] * B, lens)
    for segments in (None, 1):
        state, o = start.clone(), torch.full((T, H * dv), float("nan"), device=DEV)
        core.mlstm_scan(proj, at, ib, fb, cap, d ** -0.5, state, batch, o, heads=H, d=d, dv=dv, offset=4, segments=segments,
                        chunks=segments is None)
        assert torch.equal(state[0], start[0]) and torch.equal(state[B + 1], start[B + 1]) and torch.equal(state[:, :4], start[:, :4])
        t0 = 0
        for i, n in enumerate(lens):
            x = proj[t0:t0 + n].double()
            q, k = (x[:, at[c]:at[c] + H * d].view(n, H, d) for c in "qk")
            v = x[:, at["v"]:at["v"] + H * dv].view(n, H, dv)
            li = cap * torch.tanh((x[:, at["i"]:at["i"] + H] + ib.double()) / cap)
            lf = torch.nn.functional.logsigmoid(cap * torch.tanh((x[:, at["f"]:at["f"] + H] + fb.double()) / cap))
            S, z, m, ref = start[i + 1, 4:4 + H * d * dv].double().view(H, d, dv), norm[i + 1, 0].double().view(H, d), torch.zeros(H, device=DEV, dtype=torch.float64), []
            for t in range(n):
                new = torch.maximum(lf[t] + m, li[t])
                a, b = torch.exp(lf[t] + m - new), torch.exp(li[t] - new)
                m, S, z = new, a[:, None, None] * S + b[:, None, None] * k[t][:, :, None] * v[t][:, None], a[:, None] * z + b[:, None] * k[t]
                den = torch.maximum((z * q[t]).sum(-1).abs() * d ** -0.5, torch.exp(-m)) + 1e-6
                ref.append(torch.einsum("hdv,hd->hv", S, q[t]) * d ** -0.5 / den[:, None])
            ref, got = torch.stack(ref), o[t0:t0 + n].view(n, H, dv).double()
            # sums of up to 200 terms of size 1 over a denominator of at least e^(-m): relative to the largest output
            assert float((got - ref).abs().max()) < 3e-5 * float(ref.abs().max()), (segments, i)
            assert float((state[i + 1, 4:4 + H * d * dv].double().view(H, d, dv) - S).abs().max()) < 3e-5 * float(S.abs().max()), (segments, i)
            held = state[i + 1, 4 + H * d * dv:4 + H * d * (dv + copies)].double().view(copies, H, d)
            assert float((held - z).abs().max()) < 3e-5 * float(z.abs().max()), (segments, i)
            assert float((state[i + 1, 4 + H * d * (dv + copies):4 + floats].double() - m).abs().max()) < 1e-5 * max(1.0, float(m.abs().max()))
            t0 += n


@pytest.mark.parametrize("column", ["k", "v"])
@pytest.mark.parametrize("bad", [math.inf, math.nan])
@pytest.mark.parametrize("d,dv,n,where", [(64, 128, 200, 64), (64, 128, 200, 130), (20, 36, 64, 63), (128, 130 * 2, 70, 5)])
def test_what_a_token_brings_reaches_no_earlier_output_of_the_memory(core, column, bad, d, dv, n, where):
    H = 2
    g = torch.Generator(device=DEV).manual_seed(where)
    at = {"q": 0, "k": H * d, "v": 2 * H * d, "i": 2 * H * d + H * dv, "f": 2 * H * d + H * dv + H}
    proj = torch.randn(n, -(-(at["f"] + H) // 4) * 4, device=DEV, generator=g)
    ib, fb = torch.randn(H, device=DEV, generator=g), torch.randn(H, device=DEV, generator=g) + 2
    batch = G.make_batch(DEV, [1], [0], [n])

    def run():
        state = torch.zeros(2, -(-core.mlstm_state_floats(H, d, dv) // 4) * 4, device=DEV)
        o = torch.full((n, H * dv), 7.0, device=DEV)
        core.mlstm_scan(proj, at, ib, fb, 9.0, d ** -0.5, state, batch, o, heads=H, d=d, dv=dv, chunks=True)
        return o

    plain = run()
    proj[where, at[column]] = bad
    got = run()
    assert torch.equal(got[:where], plain[:where])
    assert not bool(got[where].isfinite().all()) and bool(plain.isfinite().all())


@pytest.mark.parametrize("chunks", [False, True])
@pytest.mark.parametrize("channel", [True, False])
@pytest.mark.parametrize("column", ["k", "v"])
@pytest.mark.parametrize("bad", [math.inf, math.nan])
@pytest.mark.parametrize("d,dv,n,where", [(128, 128, 50, 31), (128, 128, 50, 33), (12, 20, 15, 14)])
def test_what_a_token_brings_reaches_no_earlier_output_of_the_delta_rule(core, chunks, channel, column, bad, d, dv, n, where):
    H = 2
    g = torch.Generator(device=DEV).manual_seed(where)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    unit = torch.nn.functional.normalize
    qkv = torch.cat([x.reshape(n, -1) for x in (unit(r(n, H, d), dim=-1) * d ** -0.5, unit(r(n, H, d), dim=-1), r(n, H, dv))], 1).contiguous()
    step = torch.cat([torch.sigmoid(r(n, H)), torch.zeros(n, H, device=DEV) if channel else -torch.rand(n, H, device=DEV, generator=g)], 1).contiguous()
    decay = torch.rand(n, H * d, device=DEV, generator=g) if channel else None
    batch, start = G.make_batch(DEV, [1], [0], [n]), r(2, H * d * dv)

    def run():
        o = torch.full((n, H * dv), 7.0, device=DEV)
        core.delta_scan(qkv, step, start.clone(), batch, o, heads=H, kv_heads=H, d=d, dv=dv, decay=decay, chunks=chunks)
        return o

    plain = run()
    qkv[where, H * d if column == "k" else 2 * H * d] = bad
    got = run()
    assert torch.equal(got[:where], plain[:where])
    assert not bool(got[where].isfinite().all()) and bool(plain.isfinite().all())


@pytest.mark.parametrize("channel", [True, False])
@pytest.mark.parametrize("alike", [0.0, 1.0, 3.0])          # how much the keys resemble one another
@pytest.mark.parametrize("forget", [2.0, 5.0])              # decays around sigmoid(this)
def test_the_delta_rule_over_chunks_is_no_further_off_than_four_at_a_time(core, channel, alike, forget):
    H, d, dv, n = 4, 128, 64, 400
    g = torch.Generator(device=DEV).manual_seed(5)
    r = lambda *s: torch.randn(*s, device=DEV, generator=g)  # noqa: E731
    unit, soft = torch.nn.functional.normalize, torch.nn.functional.softplus
    common = alike * r(1, H, d)
    q, k, v = unit(r(n, H, d) + common, dim=-1) * d ** -0.5, unit(r(n, H, d) + common, dim=-1), r(n, H, dv)
    beta, lg = torch.sigmoid(2 * r(n, H) + 2 * (alike > 0)), -soft(r(n, H) - forget)
    decay = torch.exp(-soft(r(n, H * d) - forget)) if channel else None
    qkv = torch.cat([x.reshape(n, -1) for x in (q, k, v)], 1).contiguous()
    step = torch.cat([beta, torch.zeros_like(lg) if channel else lg], 1).contiguous()
    batch, start = G.make_batch(DEV, [1], [0], [n]), 0.1 * r(2, H * d * dv)
    S, ref = start[1].double().view(H, d, dv), []
    for t in range(n):
        S = S * (decay[t].double().view(H, d, 1) if channel else torch.exp(lg[t].double())[:, None, None])
        u = beta[t].double()[:, None] * (v[t].double() - torch.einsum("hdv,hd->hv", S, k[t].double()))
        S = S + k[t].double()[:, :, None] * u[:, None]
        ref.append(torch.einsum("hdv,hd->hv", S, q[t].double()))
    ref, off = torch.stack(ref).view(n, -1), {}
    for chunks in (False, True):
        state, o = start.clone(), torch.empty(n, H * dv, device=DEV)
        core.delta_scan(qkv, step, state, batch, o, heads=H, kv_heads=H, d=d, dv=dv, decay=decay, chunks=chunks)
        off[chunks] = [float((a.double() - b).norm() / b.norm()) for a, b in ((o, ref), (state[1], S.flatten()))]
    assert off[True][0] <= off[False][0] and off[True][1] <= off[False][1], off


@pytest.mark.parametrize("forget", [0.0, 2.5, 6.0])         # the forget gate's bias
@pytest.mark.parametrize("n", [40, 300])
def test_the_memory_over_chunks_is_no_further_off_than_four_at_a_time(core, forget, n):
    H, d, dv, cap = 16, 64, 128, 15.0
    at = {"q": 0, "k": H * d, "v": 2 * H * d, "i": 2 * H * d + H * dv, "f": 2 * H * d + H * dv + H}
    off = {None: [], 1: []}
    for seed in range(4):
        g = torch.Generator(device=DEV).manual_seed(seed)
        proj = torch.randn(n, at["f"] + H, device=DEV, generator=g)
        ib, fb = (torch.randn(H, device=DEV, generator=g) + b for b in (-0.5, forget))
        batch, x = G.make_batch(DEV, [1], [0], [n]), proj.double()
        q, k = (x[:, at[c]:at[c] + H * d].view(n, H, d) for c in "qk")
        v = x[:, at["v"]:at["v"] + H * dv].view(n, H, dv)
        li = cap * torch.tanh((x[:, at["i"]:at["i"] + H] + ib.double()) / cap)
        lf = torch.nn.functional.logsigmoid(cap * torch.tanh((x[:, at["f"]:at["f"] + H] + fb.double()) / cap))
        S, z, m, ref = torch.zeros(H, d, dv, device=DEV, dtype=torch.float64), 0.0, torch.zeros(H, device=DEV, dtype=torch.float64), []
        for t in range(n):
            new = torch.maximum(lf[t] + m, li[t])
            a, b = torch.exp(lf[t] + m - new)[:, None], torch.exp(li[t] - new)[:, None]
            m, S, z = new, a[:, None] * S + b[:, None] * k[t][:, :, None] * v[t][:, None], a * z + b * k[t]
            den = torch.maximum((z * q[t]).sum(-1).abs() * d ** -0.5, torch.exp(-m)) + 1e-6
            ref.append((torch.einsum("hdv,hd->hv", S, q[t]) * d ** -0.5 / den[:, None]).flatten())
        ref = torch.stack(ref)
        for segments in off:
            state, o = torch.zeros(2, core.mlstm_state_floats(H, d, dv), device=DEV), torch.empty(n, H * dv, device=DEV)
            core.mlstm_scan(proj, at, ib, fb, cap, d ** -0.5, state, batch, o, heads=H, d=d, dv=dv, segments=segments,
                            chunks=segments is None)
            # (a token's own relative error: where n . q cancels an output is far off in any form, and such outputs, few,
            # would decide a norm over all)
            e, r = (o.double() - ref).view(n, H, dv).norm(dim=2), ref.view(n, H, dv).norm(dim=2)
            off[segments].append(e / r)
    four, chunks = (float(torch.cat(off[s]).median()) for s in (1, None))
    # the medians of 4 x 16 x n errors are known to about 1 / sqrt(2,560) of themselves; both share what the gates' rounding brings
    assert chunks <= 1.02 * four, (chunks, four)


@pytest.mark.parametrize("d,dv", [(64, 128), (12, 260), (128, 36)])
def test_a_chunks_own_terms_of_the_memory_are_added_up_before_they_meet_the_carried_state(core, d, dv):
    """Gates of exactly 1, queries and keys along one channel: an output is (carried + own) over one denominator, where sixteen own terms are
    less than half a unit in the carried state's last place and sixty-four are several.  In 32 bits to the bit: products with
    a power of two are exact, so the sums alone round."""
    H, n = 2, 64
    at = {"q": 0, "k": H * d, "v": 2 * H * d, "i": 2 * H * d + H * dv, "f": 2 * H * d + H * dv + H}
    proj = torch.zeros(n, -(-(at["f"] + H) // 4) * 4, device=DEV)
    for h in range(H):
        proj[:, at["q"] + h * d], proj[:, at["k"] + h * d] = 1.0, 2.0 ** -10       # |n . q| <= 2^-4, so the denominator is 1 + 1e-6
    g = torch.Generator(device=DEV).manual_seed(d)
    v = 1024 * (0.05 + 0.0125 * torch.rand(n, H * dv, device=DEV, generator=g))
    proj[:, at["v"]:at["v"] + H * dv] = v
    proj[:, at["f"]:at["f"] + H] = 1e4                                             # log f = -log(1 + e^-100): f = 1
    zero = torch.zeros(H, device=DEV)
    state, o = torch.zeros(2, -(-core.mlstm_state_floats(H, d, dv) // 4) * 4, device=DEV), torch.empty(n, H * dv, device=DEV)
    state[1, :H * d * dv].view(H, d, dv)[:, 0] = 2.0 ** 24
    core.mlstm_scan(proj, at, zero, zero, 100.0, 1.0, state, G.make_batch(DEV, [1], [0], [n]), o, heads=H, d=d, dv=dv, chunks=True)
    terms, own, want = v.cpu() * 2.0 ** -10, torch.zeros(n, H * dv), torch.empty(n, H * dv)
    for t in range(n):
        for x0 in range(0, t + 1, 16):
            part = torch.zeros(H * dv)
            for x in range(x0, min(x0 + 16, t + 1)):
                part = part + terms[x]
            own[t] = own[t] + part
        want[t] = (own[t] + 2.0 ** 24) / (torch.ones(()) + torch.tensor(1e-6))
    assert float(own[15].max()) < 1.01 and float(own[63].min()) > 3 and torch.equal(o.cpu(), want)


def test_segments_asked_for_by_the_environment_reach_the_memory(core, monkeypatch):
    H, d, dv, n = 2, 64, 128, 600
    at = {"q": 0, "k": H * d, "v": 2 * H * d, "i": 2 * H * d + H * dv, "f": 2 * H * d + H * dv + H}
    g = torch.Generator(device=DEV).manual_seed(1)
    proj, ib, fb = torch.randn(n, at["f"] + H, device=DEV, generator=g), torch.zeros(H, device=DEV), torch.ones(H, device=DEV)
    batch = G.make_batch(DEV, [1], [0], [n])

    def run(segments):
        state, o = torch.zeros(2, -(-core.mlstm_state_floats(H, d, dv) // 4) * 4, device=DEV), torch.empty(n, H * dv, device=DEV)
        core.mlstm_scan(proj, at, ib, fb, 9.0, d ** -0.5, state, batch, o, heads=H, d=d, dv=dv, segments=segments)
        return o

    for n_seg in (1, 3):
        monkeypatch.setenv("MOE_B200_SCAN_SEGMENTS", str(n_seg))
        assert torch.equal(run(None), run(n_seg))


def test_short_steps_and_many_sequences_keep_the_form_of_four(core, monkeypatch):
    """A step of few tokens a sequence, or one whose blocks fill the SMs anyway, launches what it did before there were chunks."""
    H, d, dv = 16, 64, 128
    at = {"q": 0, "k": H * d, "v": 2 * H * d, "i": 2 * H * d + H * dv, "f": 2 * H * d + H * dv + H}
    taken, L = [], core.lib()
    monkeypatch.setattr(core, "lib", lambda: type("Spy", (), {"__getattr__": lambda _, name: (taken.append(name), getattr(L, name))[1]})())
    for B, n, over_chunks in ((1, 2, False), (64, 2, False), (1, 128, False), (8, 300, False), (1, 256, True), (2, 300, True)):
        proj, z = torch.randn(B * n, at["f"] + H, device=DEV), torch.zeros(H, device=DEV)
        state, o = torch.zeros(B + 1, core.mlstm_state_floats(H, d, dv), device=DEV), torch.empty(B * n, H * dv, device=DEV)
        taken.clear()
        core.mlstm_scan(proj, at, z, z, 9.0, d ** -0.5, state, G.make_batch(DEV, list(range(1, B + 1)), [0] * B, [n] * B), o, heads=H, d=d, dv=dv)
        assert ("moe_mlstm_chunks" in taken) == over_chunks, (B, n)


def test_short_steps_of_the_delta_rule_keep_the_form_of_four(core, monkeypatch):
    H, d, dv = 16, 128, 128
    asked, L = [], core.lib()
    monkeypatch.setattr(core, "lib", lambda: type("Spy", (), {"__getattr__": lambda _, name: (asked.append(name), getattr(L, name))[1]})())
    for B, n, over_chunks in ((1, 2, False), (1, 64, False), (1, 128, False), (2, 200, False), (1, 160, True)):
        qkv, step = torch.zeros(B * n, 2 * H * d + H * dv, device=DEV), torch.zeros(B * n, 2 * H, device=DEV)
        state, o = torch.zeros(B + 1, H * d * dv, device=DEV), torch.empty(B * n, H * dv, device=DEV)
        asked.clear()
        core.delta_scan(qkv, step, state, G.make_batch(DEV, list(range(1, B + 1)), [0] * B, [n] * B), o, heads=H, kv_heads=H, d=d, dv=dv)
        assert ("moe_delta_chunk_floats" in asked) == over_chunks, (B, n)


def test_a_long_delta_step_goes_window_by_window(core):
    """The scratch of the chunks is bounded; a step that needs more of it gives what its sequences give alone, to the bit."""
    H, d, dv, lens = 16, 128, 128, [3000, 517]
    T, r = sum(lens), lambda *s: torch.randn(*s, device=DEV)
    unit = torch.nn.functional.normalize
    qkv = torch.cat([x.reshape(T, -1) for x in (unit(r(T, H, d), dim=-1), unit(r(T, H, d), dim=-1), r(T, H, dv))], 1).contiguous()
    step, decay, start = torch.sigmoid(r(T, 2 * H)), torch.sigmoid(r(T, H * d) + 2), r(3, H * d * dv)
    floats = core.lib().moe_delta_chunk_floats
    assert floats(10 * T, 2, H, H, d, dv) == floats(T, 2, H, H, d, dv) <= 1 << 25 and floats(3000, 1, H, H, d, dv) < floats(T, 2, H, H, d, dv)
    run = lambda a, b, state, slots, o: core.delta_scan(  # noqa: E731
        qkv[a:b], step[a:b], state, G.make_batch(DEV, slots, [0] * len(slots), [lens[s - 1] for s in slots]), o, heads=H, kv_heads=H,
        d=d, dv=dv, decay=decay[a:b], chunks=True)
    whole, state = torch.full((T, H * dv), float("nan"), device=DEV), start.clone()
    run(0, T, state, [1, 2], whole)
    apart, one = torch.empty_like(whole), start.clone()
    run(0, 3000, one, [1], apart[:3000])
    run(3000, T, one, [2], apart[3000:])
    assert torch.equal(whole, apart) and torch.equal(state, one)


def test_a_long_step_of_the_memory_goes_window_by_window(core):
    H, d, dv, lens = 32, 128, 256, [1500, 1003]
    T, floats = sum(lens), core.lib().moe_mlstm_chunk_floats
    assert floats(20 * T, 2, H, d, dv) == floats(T, 2, H, d, dv) <= 1 << 25 and floats(1500, 1, H, d, dv) < floats(T, 2, H, d, dv)
    at = {"q": 0, "k": H * d, "v": 2 * H * d, "i": 2 * H * d + H * dv, "f": 2 * H * d + H * dv + H}
    proj, ib, fb = torch.randn(T, at["f"] + H, device=DEV), torch.randn(H, device=DEV), torch.randn(H, device=DEV) + 2
    state = torch.zeros(3, -(-core.mlstm_state_floats(H, d, dv) // 4) * 4, device=DEV)
    one = state.clone()
    run = lambda a, b, st, slots, o: core.mlstm_scan(  # noqa: E731
        proj[a:b], at, ib, fb, 9.0, d ** -0.5, st, G.make_batch(DEV, slots, [0] * len(slots), [lens[s - 1] for s in slots]), o,
        heads=H, d=d, dv=dv, chunks=True)
    whole, apart = torch.full((T, H * dv), float("nan"), device=DEV), torch.empty(T, H * dv, device=DEV)
    run(0, T, state, [1, 2], whole)
    run(0, 1500, one, [1], apart[:1500])
    run(1500, T, one, [2], apart[1500:])
    assert torch.equal(whole, apart) and torch.equal(state, one)


def test_a_stack_of_no_weights_leaves_the_rows_alone(core):
    st, out = core.new_status(DEV), torch.full((5, 8), 3.0, device=DEV)
    core.gemm_generic(torch.ones(5, 16, device=DEV), torch.empty(0, 8, 16, device=DEV), out, group_offsets=torch.zeros(1, dtype=torch.int32, device=DEV),
                      status=st)
    assert bool((out == 3).all()) and int(st[0]) == 0


@pytest.mark.parametrize("counts,before,after", [([40, 0, 70], 7, 5), ([3, 2], 4, 6), ([20, 300], 1, 0)])
def test_rows_of_no_group_are_left_alone(core, counts, before, after):
    torch.manual_seed(before)
    E, N, K, M = len(counts), 132, 772, before + sum(counts) + after
    a, w, st = torch.randn(M, K, device=DEV), torch.randn(E, N, K, device=DEV), core.new_status(DEV)
    offs = torch.tensor(np.cumsum([before] + counts), dtype=torch.int32, device=DEV)
    out = torch.full((M, N), 7.0, device=DEV)
    core.gemm_generic(a, w, out, group_offsets=offs, status=st)
    assert bool((out[:before] == 7).all()) and bool((out[M - after:] == 7).all())
    for g in range(E):
        x = a[offs[g]:offs[g + 1]]
        assert bool(((out[offs[g]:offs[g + 1]].double() - x.double() @ w[g].double().T).abs() <= bound(x, w[g])).all()), g
    assert int(st[0]) == 0


@pytest.mark.parametrize("M,N,K", [(1152, 2048, 5632), (520, 3584, 20480), (333, 6145, 4100)])
def test_the_sums_of_k_splits_find_room(core, M, N, K):
    """The chunks' sums of K splits take 128 MB at most: a product that would need more goes over its rows in passes.  The result is
    the same to the bit as its rows' alone."""
    torch.manual_seed(M)
    assert all(core.lib().moe_gemm_scratch_floats(m, N, K, 0) <= 1 << 25 for m in range(1, 4 * M, 7))
    a, w, st = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV), core.new_status(DEV)
    out = torch.full((M + 1, N), float("nan"), device=DEV)
    core.gemm_generic(a, w, out[:M], status=st)
    few = torch.empty(8, N, device=DEV)
    for r in (0, M // 2, M - 8):
        core.gemm_generic(a[r:r + 8], w, few, status=st)
        assert torch.equal(few, out[r:r + 8]), r
    assert bool(out[M].isnan().all()) and int(st[0]) == 0


@pytest.mark.parametrize("tile,split,blocks", [(128, 0, 2), (128, 1, 2), (64, 0, 3), (64, 1, 3), (32, 0, 5), (32, 1, 6)])
def test_an_sm_holds_the_blocks_the_plan_counts_with(core, tile, split, blocks):
    assert core.lib().moe_gemm_tile_room(tile, split) >= blocks


@pytest.mark.parametrize("hd", [128, 64])
@pytest.mark.parametrize("before,new,window,keep,where", [(0, 256, None, 0, 100), (0, 256, None, 0, 200), (70, 300, None, 0, 140), (0, 400, 50, 0, 10),
                                                          (0, 400, 50, 0, 150), (37, 290, 130, 70, 90)])
def test_a_value_reaches_no_query_of_another_tile_that_does_not_see_it(core, hd, before, new, window, keep, where):
    """An infinite or NaN value of one key: the queries of a tile of 64 none of which sees the key are the same to the bit."""
    from moe_b200.cache import KVCache, KVRequest

    torch.manual_seed(where)
    T = before + new
    cache = KVCache({0: KVRequest(1, hd, window, keep=keep) if keep else KVRequest(1, hd, window)}, {0: None}, max_tokens=64 * 30, max_slots=2,
                    dtype=torch.float32, device=DEV)
    view, slot, st = cache.view(0), cache.acquire(), core.new_status(DEV)
    K, V, q = torch.randn(T, 1, hd, device=DEV), torch.randn(T, 1, hd, device=DEV), torch.randn(new, 1, hd, device=DEV)
    if before:
        G.give_pages(cache, slot, before)
        core.kv_commit(K[:before].contiguous(), V[:before].contiguous(), view, G.make_batch(DEV, [slot], [0], [before]), st)
    G.give_pages(cache, slot, T)
    batch, outs = G.make_batch(DEV, [slot], [before], [new]), []
    assert where >= before
    for bad in (None, math.inf, math.nan):
        vn = V[before:].clone()
        if bad is not None:
            vn[where - before] = bad
        outs.append(torch.empty(new, hd, device=DEV))
        assert core.attention_tiled(q, K[before:].contiguous(), vn, view, batch, outs[-1], nh=1, window=window, scale=hd ** -0.5, use_local=True,
                                    status=st, keep=keep)
    clean = 0
    for r0 in range(0, new, 64):
        p = torch.arange(before + r0, before + min(r0 + 64, new))
        lo = (p + 1 - window).clamp(min=0) if window else torch.zeros_like(p)
        if not bool(((where <= p) & ((where >= lo) | (where < keep))).any()):
            clean += 1
            assert torch.equal(outs[1][r0:r0 + 64], outs[0][r0:r0 + 64]) and torch.equal(outs[2][r0:r0 + 64], outs[0][r0:r0 + 64]), r0
    assert clean > 0 and not bool(outs[1].isfinite().all()) and bool(outs[0].isfinite().all()) and int(st[0]) == 0


def form(core, M, N, K, groups=0):
    import ctypes

    out = (ctypes.c_int * 5)()
    core.lib().moe_gemm_plan(M, N, K, groups, ctypes.addressof(out))
    return list(out)             # rows a tile of the form for few rows (or 0), rows a tile, K splits, chunks a split, rows a pass


# one size for every form on 148 SMs: (rows a tile, with K splits or not, chunks a split more than one or not)
@pytest.mark.parametrize("M,N,K,tile,split,several", [
    (4921, 6145, 2052, 128, False, True), (4920, 2048, 2048, 64, False, True), (640, 6144, 2048, 128, False, True),
    (512, 2048, 5632, 128, True, True), (200, 2048, 2048, 128, True, False), (100, 6145, 2052, 128, True, True),
    (300, 2048, 2048, 64, True, True), (40, 6144, 2048, 64, True, False), (400, 2049, 2044, 32, True, True),
    (17, 11264, 2048, 32, True, False), (1152, 2047, 5632, 64, True, True)])
def test_every_tile_form_gives_the_same_bits(core, M, N, K, tile, split, several):
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        rows, t, splits, per, _ = form(core, M, N, K)
        assert rows == 0 and (t, splits > 1, per > 1) == (tile, split, several), (t, splits, per)
    torch.manual_seed(M + N)
    a, w, b, st = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV), torch.randn(N, device=DEV), core.new_status(DEV)
    out = torch.full((M + 1, N), float("nan"), device=DEV)
    core.gemm_generic(a, w, out[:M], bias=b, status=st)
    assert bool(out[M].isnan().all())
    some = torch.tensor(sorted({0, 1, 31, 32, 63, 64, 127, 128, M // 2, M - 2, M - 1} & set(range(M))), device=DEV)
    ref = a[some].double() @ w.double().T + b.double()
    assert bool(((out[some].double() - ref).abs() <= bound(a[some], w) + 2 * EPS * ref.abs()).all())
    few = torch.empty(1, N, device=DEV)
    for r in some.tolist():
        core.gemm_generic(a[r:r + 1], w, few, bias=b, status=st)
        assert torch.equal(few, out[r:r + 1]), r
    assert int(st[0]) == 0


@pytest.mark.parametrize("G,each,N,K,tile,splits", [(24, 20, 1284, 516, 32, 3), (24, 24, 1284, 516, 64, 2), (24, 40, 1410, 516, 64, 1),
                                                    (24, 90, 1284, 772, 128, 1), (60, 40, 2816, 516, 32, 1), (24, 600, 1284, 516, 128, 1)])
def test_every_tile_form_of_many_groups(core, G, each, N, K, tile, splits):
    """Several hundred blocks and more; groups of unequal size, empty ones among them."""
    counts = [0 if g % 7 == 3 else each + (g * 37) % (each + 1) - each // 2 for g in range(G)]
    M = sum(counts)
    if torch.cuda.get_device_properties(0).multi_processor_count == 148:
        assert form(core, M, N, K, G)[:3] == [0, tile, splits], form(core, M, N, K, G)
    torch.manual_seed(G + each)
    a, w, st = torch.randn(M, K, device=DEV), torch.randn(G, N, K, device=DEV), core.new_status(DEV)
    offs = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32, device=DEV)
    out, few = torch.full((M + 1, N), float("nan"), device=DEV), torch.empty(1, N, device=DEV)
    core.gemm_generic(a, w, out[:M], group_offsets=offs, status=st)
    assert bool(out[M].isnan().all())
    for g in range(0, G, max(1, G // 8)):
        if counts[g]:
            x = a[offs[g]:offs[g + 1]]
            assert bool(((out[offs[g]:offs[g + 1]].double() - x.double() @ w[g].double().T).abs() <= bound(x, w[g])).all()), g
            for r in {0, counts[g] // 2, counts[g] - 1}:
                core.gemm_generic(x[r:r + 1], w[g], few, status=st)
                assert torch.equal(few[0], out[int(offs[g]) + r]), (g, r)
    assert int(st[0]) == 0
