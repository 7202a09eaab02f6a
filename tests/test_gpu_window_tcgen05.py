"""The window attention of prompts with keys and values of 64 or 128 columns (tcgen05) against the in-order warp kernel, which
holds everything in 32-bit: windows, chunks, kept first keys, sinks and gates, rows that end inside a tile, requests side by
side, and values that are not finite."""
from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
HEADS, KV, PAGE = 4, 2, 24                                   # (pages that are no power of two)


@pytest.fixture(scope="module")
def ops():
    from pih_b200.kernels import get_ops
    return get_ops(torch.device(DEV))


def _case(dim, vdim, requests, seed):
    """requests: (earlier tokens, rows) of each; the cache holds every request's tokens, pages out of order."""
    g = torch.Generator(DEV).manual_seed(seed)
    normal = lambda *s: torch.randn(*s, generator=g, device=DEV).to(torch.bfloat16)
    width = max(-(-(past + n) // PAGE) for past, n in requests)
    pages = width * len(requests)
    table = torch.randperm(pages, generator=torch.Generator().manual_seed(seed)).to(torch.int32).reshape(len(requests), width)
    cache = normal(pages, PAGE, KV * (dim + vdim))
    cu = [0]
    for _, n in requests:
        cu.append(cu[-1] + n)
    t = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)
    starts = [past for past, _ in requests]
    step = SimpleNamespace(positions=t([past + i for past, n in requests for i in range(n)]),
                           request_of_row=t([r for r, (_, n) in enumerate(requests) for _ in range(n)]), cu_q=t(cu),
                           num_requests=len(requests), host_cu_q=cu, host_q_start=starts, q_start=t(starts), meta=None,
                           attention_plans=None)
    return dict(q=normal(cu[-1], HEADS * dim), cache=cache, block_table=table.to(DEV), step=step, heads=HEADS, kv_heads=KV,
                key_dim=dim, value_dim=vdim, scale=dim ** -0.5, softcap=0.0, bias=None), normal


def _both(ops, case, **options):
    q = case.pop("q")
    got = ops.window_attention(q, **case, **options)
    ops.window_attention_fast = False
    try:
        want = ops.window_attention(q, **case, **options)
    finally:
        del ops.window_attention_fast
    ops.check_errors()
    return got.float(), want.float()


@pytest.mark.parametrize("dim,vdim", [(64, 64), (64, 128), (128, 64), (128, 128)])
@pytest.mark.parametrize("requests", [[(0, 17)], [(0, 128)], [(63, 129)], [(0, 300), (500, 1), (100, 40)], [(1000, 257)]])
@pytest.mark.parametrize("rule", [dict(window=0, keep_first=0), dict(window=1, keep_first=0), dict(window=100, keep_first=0),
                                  dict(window=130, keep_first=70), dict(window=0, keep_first=3, chunk=96)])
def test_against_the_warp_kernel(ops, dim, vdim, requests, rule):
    case, normal = _case(dim, vdim, requests, seed=dim + vdim + len(requests))
    rows = case["q"].shape[0]
    sink = normal(HEADS).float() if rule["window"] else None
    gate_per = "column" if rule.get("chunk") else "head"
    gate = normal(rows, HEADS * vdim)
    got, want = _both(ops, case, sink=sink, gate=gate, gate_per=gate_per, **rule)
    # both round once to bf16 (2^-9 of the value); the weights' pairs are 2^-17 off and so are their sums
    scale = float(want.abs().max())
    torch.testing.assert_close(got, want, rtol=2.0 ** -7, atol=scale * 2.0 ** -14)


@pytest.mark.parametrize("value", [float("nan"), float("inf")])
def test_a_value_that_is_not_finite_reaches_the_rows_that_see_it_alone(ops, value):
    dim, n, at, window = 128, 300, 150, 60
    case, _ = _case(dim, dim, [(0, n)], seed=5)
    flat = case["block_table"][0, at // PAGE], at % PAGE
    clean = dict(case, cache=case["cache"].clone())
    clean["cache"][flat][KV * dim:] = 0
    case["cache"][flat][KV * dim + 7] = value                # one value column of the first key/value head
    options = dict(window=window, keep_first=0, sink=None, gate=None)
    got = ops.window_attention(case.pop("q"), **case, **options).float().reshape(n, HEADS, dim)
    want = ops.window_attention(clean.pop("q"), **clean, **options).float().reshape(n, HEADS, dim)
    ops.clear_errors()
    sees = torch.zeros(n, dtype=torch.bool, device=DEV)
    sees[at:at + window] = True
    assert torch.isfinite(got[~sees]).all() and torch.isfinite(got[:, HEADS // KV:]).all()
    torch.testing.assert_close(got[~sees], want[~sees], rtol=2.0 ** -7, atol=2.0 ** -12)
    assert not torch.isfinite(got[sees][:, :HEADS // KV, 7]).any()
    seen_others = got[sees][:, :HEADS // KV, torch.arange(dim, device=DEV) != 7]
    assert torch.isfinite(seen_others).all()
