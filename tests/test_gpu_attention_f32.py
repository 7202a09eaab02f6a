"""The 32-bit attention of head sizes 64 and 128: edges of its key tiles and row groups against float64, and that a cut or
the batch changes no bit."""
import math

import pytest
import torch

from test_gpu_kernels import _attention_reference, _paged_setup

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from pih_b200.kernels import get_ops
    return get_ops(torch.device("cuda:0"))


def _run(ops, s, rows, heads, kv_heads, D, window):
    return ops.paged_attention_generic(s["q"][rows], heads=heads, kv_heads=kv_heads, head_dim=D, kv_cache=s["cache"],
                                       block_table=s["table"], request_of_row=s["req_of_row"][rows],
                                       positions=s["positions"][rows], scale=1 / math.sqrt(D), window=window or 0)


@pytest.mark.parametrize("heads,kv_heads,D", [(4, 2, 128), (16, 1, 64), (3, 3, 128), (14, 2, 64), (5, 1, 128)])
@pytest.mark.parametrize("lens,new,window", [([1, 31, 32, 33], [1, 31, 2, 33], None), ([129, 700, 128], [129, 3, 1], None),
                                             ([300, 97], [40, 1], 33), ([90, 64], [17, 64], 1)])
def test_against_float64(ops, heads, kv_heads, D, lens, new, window):
    s = _paged_setup(torch.float32, lens, new, heads, kv_heads, D, 16, seed=21)
    out = _run(ops, s, slice(None), heads, kv_heads, D, window)
    ops.check_errors()
    torch.testing.assert_close(out.cpu().double(), _attention_reference(s, lens, new, 1 / math.sqrt(D), window),
                               rtol=2e-5, atol=2e-6)
    for lo, hi in ((0, 1), (1, 20), (20, sum(new)), (sum(new) - 1, sum(new))):      # rows alone and cut otherwise
        assert torch.equal(_run(ops, s, slice(lo, hi), heads, kv_heads, D, window), out[lo:hi])


def test_rows_of_padding_and_keys_without_a_page(ops):
    s = _paged_setup(torch.float32, [70, 40], [4, 2], 4, 2, 128, 16, seed=5)
    whole = _run(ops, s, slice(None), 4, 2, 128, None)
    s["req_of_row"][4:] = -1                                                         # rows of no request stay out of it
    assert torch.equal(_run(ops, s, slice(None), 4, 2, 128, None)[:4], whole[:4])
    ops.check_errors()
    s["table"][0, 1] = -1
    _run(ops, s, slice(None), 4, 2, 128, None)
    with pytest.raises(Exception):
        ops.check_errors()
    ops.clear_errors()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("heads,kv_heads", [(4, 4), (4, 2), (16, 1)])
@pytest.mark.parametrize("n,window", [(40, None), (17, None), (150, 20), (33, 1)])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
def test_values_that_a_row_does_not_see(ops, D, heads, kv_heads, n, window, value):
    """A value that is infinite or no number reaches the rows that see its key; the bits of earlier rows of the same blocks, and
    of rows whose window has left it behind, stay."""
    s = _paged_setup(torch.float32, [n], [n], heads, kv_heads, D, 16, seed=n)
    whole = _run(ops, s, slice(None), heads, kv_heads, D, window)
    kinds = {"value": 1} if value != value else {"value": 1, "key": 0}        # (a key of NaN or infinity spoils its rows' sums)
    for at in {0, 5, n // 2, n - 1}:
        for kind in kinds.values():
            page = int(s["table"][0, at // 16])
            kept = s["cache"][page, kind, 0, at % 16, 3].clone()
            s["cache"][page, kind, 0, at % 16, 3] = value
            got = _run(ops, s, slice(None), heads, kv_heads, D, window)
            s["cache"][page, kind, 0, at % 16, 3] = kept
            blind = [t for t in range(n) if t < at or (window and t >= at + window)]
            assert torch.equal(got[blind], whole[blind])
            if kind == 1:
                sees = [t for t in range(n) if t not in blind]
                assert not bool(got[sees][:, 3].isfinite().any())
            ops.clear_errors()
