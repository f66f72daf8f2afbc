"""The forms of the 32-bit kernels that a size picks, at the sizes where they meet: products of few and of many rows
(16-byte operands; the tile heights; group counts), against float64."""
import numpy as np
import pytest
import torch

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
