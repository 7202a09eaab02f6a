"""The 32-bit product in tiles: remainders of every edge, sliced k, batches and views, against sums in 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from pih_b200.kernels import get_ops
    return get_ops(torch.device("cuda:0"))


def _bound(x, w):
    # a chain of 16 products, at most a dozen tiles of 32 in a slice and eight slices: every product meets fewer than 64
    # roundings of 2^-24 of a sum that is at most the sum of the magnitudes
    return 64 * 2.0 ** -24 * (x.double().abs() @ w.double().abs().T)


@pytest.mark.parametrize("M", [1, 8, 9, 32, 33, 65, 200])
@pytest.mark.parametrize("N,K", [(64, 4), (61, 36), (130, 508), (200, 512), (65, 1028), (1024, 2052), (300, 3072)])
def test_tiles(ops, M, N, K):
    gen = torch.Generator("cuda").manual_seed(M * 7919 + N * 31 + K)
    x = torch.randn(M, K + 8, device="cuda", generator=gen)[:, 4:4 + K]          # a view: rows wider apart than K
    w = torch.randn(N, K, device="cuda", generator=gen)
    got, want = ops.linear(x, w), x.double() @ w.double().T
    assert ((got.double() - want).abs() <= _bound(x, w)).all()
    few = ops.linear(x[-1:].clone(), w)                                           # neither the batch nor the tile matters
    assert torch.equal(few[0], got[-1])


def test_unaligned_views_and_batches(ops):
    gen = torch.Generator("cuda").manual_seed(3)
    x, w = torch.randn(40, 1031, device="cuda", generator=gen), torch.randn(70, 1026, device="cuda", generator=gen)
    for a, b in ((x[:, 1:1025], w[:, :1024]), (x[:, 4:1030], w)):
        assert ((ops.linear(a, b).double() - a.double() @ b.double().T).abs() <= 2 * _bound(a, b)).all()
    xb, wb = torch.randn(37, 3, 192, device="cuda", generator=gen), torch.randn(3, 128, 192, device="cuda", generator=gen)
    got = ops.linear_batched(xb, wb)
    for b in range(3):
        assert ((got[:, b].double() - xb[:, b].double() @ wb[b].double().T).abs() <= _bound(xb[:, b], wb[b])).all()
