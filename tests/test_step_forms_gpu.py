"""The kernels and forms of a step that a size or a pitch picks, at the sizes where they meet."""
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
