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
