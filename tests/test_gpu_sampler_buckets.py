"""Sampling by buckets and what is left to the radix passes: every choice is the first place of the sorted order where the
cumulative share passes the draw, in float64."""
import numpy as np
import pytest
import torch

import plain_impl
from test_gpu_kernels import _sample_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from pih_b200.kernels import get_ops
    return get_ops(torch.device("cuda:0"))


@pytest.mark.parametrize("vocab", [7, 1983, 32768, 151936])
@pytest.mark.parametrize("shape", ["normal", "equal", "two plateaus", "far apart", "one high", "levels", "levels and masked", "cold", "narrow", "very narrow"])
def test_choices(ops, vocab, shape):
    g = torch.Generator().manual_seed(vocab)
    logits = torch.randn(12, vocab, generator=g) * 2.5
    if shape == "equal":
        logits[:] = -3.25
    if shape == "two plateaus":                                  # more equal values than a bucket's list holds
        logits = torch.where(logits > 0.1, 4.0, -1.0)
    if shape == "far apart":                                     # most masses are zero; a top_k ends among them
        logits *= 100.0
    if shape.startswith("levels"):                               # of a quarter each; more equal values than a list holds
        logits = torch.round(logits * 2) / 4
    if shape == "levels and masked":
        logits[:, ::3] = -1e9
    if shape == "cold":                                          # as 0.1 would make of them: a top_k ends beyond all mass
        logits *= 10.0
    if shape.endswith("narrow"):                                 # one logit above a bulk: more in a bucket than a list holds
        logits *= 0.12 if shape == "narrow" else 1e-4
        logits[:, vocab // 2] = 12.0
    if shape == "one high":
        logits[:, vocab // 2] = 60.0
    rows = [([0.7, 1.0, 2.0][i % 3], [1.0, 0.9, 0.3, 1.0][i % 4], [None, 1, 40, vocab // 2 + 1][i % 4], 5 + i, i,
             [vocab - 1] if i == 5 else []) for i in range(12)]
    got = _sample_rows(ops, logits.cuda(), rows)
    ops.check_errors()
    for i, (t, p, k, seed, ordinal, sup) in enumerate(rows):
        scaled = (logits[i].numpy() / np.float32(t)).astype(np.float32).astype(np.float64)
        order = np.lexsort((np.arange(vocab), -scaled))
        order = order[~np.isin(order, sup)][:k]
        w = np.exp(scaled[order] - scaled[order[0]])
        share = np.cumsum(w) / w.sum()
        # the 2^-44 steps and the 32-bit exponential's error (two ulps) move a boundary by less than 1e-6 of the mass; so
        # top_p may end at either side of a boundary that near, and the draw at either side of another
        u = (plain_impl.sample([0.0], temperature=1.0, top_p=1.0, top_k=None, seed=seed, ordinal=ordinal, suppressed=[])[2] + 0.5) / 2.0 ** 32
        j = int(np.nonzero(order == got[i])[0][0])
        fits = []
        for end in {int(np.searchsorted(share, p + d)) for d in (-1e-6, 0.0, 1e-6)} if p < 1.0 else {len(order) - 1}:
            kept = w[:min(end, len(order) - 1) + 1]
            cum = np.concatenate([[0.0], np.cumsum(kept) / kept.sum()])
            fits.append(j < len(kept) and cum[j] - 2e-6 <= u < cum[j + 1] + 2e-6)
        assert any(fits), (i, rows[i], got[i], j, u)
