"""Which form a tensor-core product takes by its number of rows: tiles of 64 with K splits between the few rows of a decode step
and the persistent form, pairs of CTAs from some thousand rows on.  Sizes at the edges of tiles, splits and of the rules."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.fixture
def tc():
    from moe_b200.ops import tc as t

    before = t.lib().moe_tc_set_pair(-1)
    yield t
    t.lib().moe_tc_set_pair(before)


def bound(x, w):
    """Products of bfloat16 numbers are exact in 32 bits; K of them are added, every sum off by at most one unit."""
    return (x.shape[1] + 8) * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T) + 1e-30


@pytest.mark.parametrize("M", [65, 80, 127, 128, 129, 200, 256, 257, 320, 511, 512, 513])
@pytest.mark.parametrize("N,K", [(136, 72), (2048, 2048), (256, 5632), (5000, 264)])
def test_rows_between(tc, M, N, K):
    from moe_b200.ops import core

    torch.manual_seed(M + N)
    st, x, w = core.new_status(DEV), torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N, K, device=DEV).bfloat16()
    b = torch.randn(N, device=DEV)
    for beside in (False, True):
        out = torch.full((M + 1, N), float("nan"), device=DEV)
        assert tc.gemm_tc(x, w, out[:M], bias=b, status=st, beside=beside)
        ref = x.double() @ w.double().T + b.double()
        assert bool(((out[:M].double() - ref).abs() <= bound(x, w) + 2.0 ** -23 * ref.abs()).all()) and bool(out[M].isnan().all())
    assert int(st[0]) == 0


def test_splits_between_find_room():
    from moe_b200.ops.tc import mid_splits

    for M in range(65, 1200, 7):
        for n_tiles in (1, 2, 16, 28, 36, 48, 88):
            for kb in (1, 3, 22, 32, 56, 88, 320):
                s, tiles = mid_splits(M, n_tiles, kb, 148), -(-M // 64) * n_tiles
                assert (s == 0) == (tiles > 296 or M > 512)
                assert s == 0 or (1 <= s <= 8 and tiles * s <= 296 and (s == 1 or kb // s >= 4))


@pytest.mark.parametrize("M", [3071, 3072, 4095, 4097])
@pytest.mark.parametrize("swiglu", [False, True])
def test_pairs_by_rows(tc, M, swiglu):
    from moe_b200.ops import core

    torch.manual_seed(M)
    N, K = 208, 200
    st, x, w = core.new_status(DEV), torch.randn(M, K, device=DEV).bfloat16(), torch.randn(N * (2 if swiglu else 1), K, device=DEV).bfloat16()
    out = torch.full((M, N), float("nan"), device=DEV)
    assert tc.gemm_tc(x, w, out, swiglu=swiglu, status=st)
    ref, off = x.double() @ w.double().T, bound(x, w)
    if swiglu:
        # |d silu| <= 1.1 |d gate|, then the rounding of silu (a few units) and of the product
        gate, up = ref[:, :N], ref[:, N:]
        off = 1.1 * off[:, :N] * (up.abs() + off[:, N:]) + gate.abs() * off[:, N:] + 2.0 ** -20 * (gate * up).abs()
        ref = torch.nn.functional.silu(gate) * up
    assert bool(((out.double() - ref).abs() <= off + 2.0 ** -23 * ref.abs()).all())
    assert int(st[0]) == 0


@pytest.mark.parametrize("counts", [[300, 0, 470], [256, 257, 255], [1, 900, 0, 513], [200, 200]])
@pytest.mark.parametrize("swiglu", [False, True])
def test_pairs_of_groups(tc, counts, swiglu):
    from moe_b200.ops import core

    torch.manual_seed(sum(counts))
    N, K, E, M = 176, 136, len(counts), sum(counts)
    st, x = core.new_status(DEV), torch.randn(M, K, device=DEV).bfloat16()
    w = torch.randn(E, N * (2 if swiglu else 1), K, device=DEV).bfloat16()
    offs = torch.tensor(np.concatenate([[0], np.cumsum(counts)]), dtype=torch.int32, device=DEV)
    out = torch.full((M, N), float("nan"), device=DEV)
    assert tc.gemm_tc(x, w, out, swiglu=swiglu, group_offsets=offs, status=st)
    at = 0
    for e, n in enumerate(counts):
        r = x[at:at + n].double() @ w[e].double().T
        off = bound(x[at:at + n], w[e])
        if swiglu:
            g, u = r[:, :N], r[:, N:]
            off = 1.1 * off[:, :N] * (u.abs() + off[:, N:]) + g.abs() * off[:, N:] + 2.0 ** -20 * (g * u).abs()
            r = torch.nn.functional.silu(g) * u
        assert bool(((out[at:at + n].double() - r).abs() <= off + 2.0 ** -23 * r.abs()).all()), e
        at += n
    assert int(st[0]) == 0


def test_a_token_is_routed_alike_in_a_short_and_in_a_long_prompt():
    """The router's logits, from which picks and weights are formed, are the same to the bit for any number of tokens that the
    tensor-core form takes."""
    import moe_b200
    from moe_b200.parts.base import Activations

    H = 2048
    cfg = dict(architectures=["Qwen2MoeForCausalLM"], model_type="qwen2_moe", num_hidden_layers=1, hidden_size=H, num_attention_heads=1,
               num_key_value_heads=1, head_dim=128, num_experts=60, num_experts_per_tok=4, moe_intermediate_size=16,
               shared_expert_intermediate_size=16, norm_topk_prob=False, decoder_sparse_step=1, intermediate_size=16, vocab_size=64)
    model = moe_b200.random_model(cfg, seed=0, dtype="bfloat16", device=DEV)
    part = model.blocks[0].ffn
    x = torch.randn(4500, H, device=DEV)
    short, *longer = [part.route(model.rt, Activations(act=x[:T].bfloat16(), f32=x[:T].contiguous()), None) for T in (300, 2048, 2100, 4500)]
    for got in longer:
        assert all(torch.equal(a, b[:300]) for a, b in zip(short, got))


@pytest.mark.parametrize("on_a_side_stream", [True, False])
def test_the_shared_experts_product_keeps_to_few_sms_only_beside_others(on_a_side_stream, monkeypatch):
    import moe_b200
    from moe_b200.ops import tc

    cfg = dict(architectures=["Qwen2MoeForCausalLM"], model_type="qwen2_moe", num_hidden_layers=1, hidden_size=128, num_attention_heads=1,
               num_key_value_heads=1, head_dim=128, num_experts=4, num_experts_per_tok=2, moe_intermediate_size=64,
               shared_expert_intermediate_size=256, norm_topk_prob=False, decoder_sparse_step=1, intermediate_size=16, vocab_size=64)
    model = moe_b200.random_model(cfg, seed=0, dtype="bfloat16", device=DEV)
    model.blocks[0].ffn.shared_beside = on_a_side_stream
    product, seen = tc.gemm_tc, []

    def spy(x, w, out, **k):
        if w.shape == (128, 256):
            seen.append((x.shape[0], k["beside"]))
        return product(x, w, out, **k)

    monkeypatch.setattr(tc, "gemm_tc", spy)
    eng = moe_b200.Engine(model, max_tokens=2048, max_slots=2)
    for n in (200, 512):
        slot = eng.new_sequence()
        eng.step([slot], [[1] * n], check=True)
        eng.release(slot)
    assert set(seen) == {(256, on_a_side_stream), (512, False)}


def test_branches_beside_one_another_do_not_spread_over_all_sms(monkeypatch):
    """The two mixers of a layer run side by side: from 257 rows on their products keep to the SMs they need.  The other layers' do not."""
    import kulanex_util
    import moe_b200
    from moe_b200.ops import tc

    cfg = {"architecture": "Kulanex", "vocab": 64, "width": 128, "norm": {"eps": 1e-5}, "residual_mult": 0.5,
           "layers": [kulanex_util.layer(kulanex_util.parallel(2, 1, 64, 3, 16, size=64, keep=5, rheads=2, rdim=16, rvdim=32), 0),
                      kulanex_util.layer(kulanex_util.delta(2, 2, 16, 32, 4), 0)]}
    model = moe_b200.random_model(cfg, seed=0, dtype="bfloat16", device=DEV)
    product, seen = tc.gemm_tc, []

    def spy(x, w, out, **k):
        seen.append((x.shape[0], bool(k.get("beside"))))
        return product(x, w, out, **k)

    monkeypatch.setattr(tc, "gemm_tc", spy)
    eng = moe_b200.Engine(model, max_tokens=2048, max_slots=2)
    for n, rows, marked in ((200, 256, False), (300, 512, True)):
        seen.clear()
        slot = eng.new_sequence()
        eng.step([slot], [[1] * n], check=True)
        eng.release(slot)
        of_rows = [b for r, b in seen if r == rows]
        assert any(of_rows) == marked and not all(of_rows), (n, seen)


def test_a_prompt_of_more_than_4096_tokens_is_the_same_with_and_without_pairs(tc):
    """A whole step under the default rule: a pair's products add the same terms in the same order."""
    import moe_b200

    cfg = dict(architectures=["Qwen2MoeForCausalLM"], model_type="qwen2_moe", num_hidden_layers=2, hidden_size=256, num_attention_heads=2,
               num_key_value_heads=2, head_dim=128, num_experts=4, num_experts_per_tok=2, moe_intermediate_size=128,
               shared_expert_intermediate_size=512, norm_topk_prob=False, decoder_sparse_step=1, intermediate_size=16, vocab_size=128)
    model = moe_b200.random_model(cfg, seed=0, dtype="bfloat16", device=DEV)
    eng = moe_b200.Engine(model, max_tokens=5120, max_slots=2)
    logits = []
    for pairs in (-1, 0):
        tc.lib().moe_tc_set_pair(pairs)
        slot = eng.new_sequence()
        logits.append(eng.step([slot], [[(i * 7 + 3) % 128 for i in range(4300)]], check=True).clone())
        eng.release(slot)
    assert torch.equal(*logits) and bool(logits[0].isfinite().all())
