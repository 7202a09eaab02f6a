"""Recurrences that take a prompt chunk by chunk, against their definition in float64 — remainders of a chunk, requests that go
token by token and requests of padding beside them, a state carried in — and against the token loop's own error."""
import pytest
import torch

from test_gpu_tuganex import DEV, F64, _ops, _step

pytestmark = pytest.mark.gpu


def _requests(lens):
    """A step of these requests in slots 1, 2, ..., one of padding in front of the last."""
    cu, slots = [0], []
    for i, n in enumerate(lens):
        if i == len(lens) - 1:
            cu.append(cu[-1])
            slots.append(-1)
        cu.append(cu[-1] + n)
        slots.append(i + 1)
    rows = cu[-1]
    return _step(list(range(rows)), [0] * rows, cu, slots), [(cu[i], cu[i + 1], s) for i, s in enumerate(slots) if s >= 0]


@pytest.mark.parametrize("dim, vdim", [(64, 64), (128, 128), (64, 128), (128, 192)])
@pytest.mark.parametrize("lens", [[65], [64, 128], [130, 1, 17, 16, 200], [700]])
def test_retention(dim, vdim, lens):
    ops, heads = _ops(), 3
    step, places = _requests(lens)
    T = sum(lens)
    g = torch.Generator().manual_seed(dim + T)
    qk = torch.randn(T, 2 * heads * dim, generator=g).bfloat16().to(DEV)
    v = torch.randn(T, heads * vdim + 8, generator=g).bfloat16().to(DEV)[:, 8:]
    freq = torch.tensor([1000.0 ** (-2.0 * i / 32) for i in range(16)], dtype=torch.float32, device=DEV)
    decays = torch.tensor([1.0, 0.99, 0.03], dtype=F64)
    first = torch.randn(len(lens) + 2, heads * dim * vdim, generator=g).to(DEV)
    results = []
    for chunked in (True, False):
        state, ops.chunk_min_rows = first.clone(), 64 if chunked else 1 << 30
        o = ops.retention(qk, v, frequencies=freq, decay_minus_one=(decays - 1.0).float().to(DEV), key_scale=0.25, state=state,
                          step=step, heads=heads, key_dim=dim, value_dim=vdim)
        results.append((o, state))
    ops.chunk_min_rows = type(ops).chunk_min_rows
    ops.check_errors()
    ang = torch.arange(T, device=DEV, dtype=torch.float32)[:, None] * freq                  # (angles are formed in 32 bits)
    c, s = torch.cos(ang.double())[:, None], torch.sin(ang.double())[:, None]

    def turned(x):
        a, b = x[..., :16], x[..., 16:32]
        return torch.cat([a * c - b * s, b * c + a * s, x[..., 32:]], -1)
    q, k = (turned(x.double().view(T, heads, dim)) for x in qk.chunk(2, 1))
    k, vv, gamma = 0.25 * k, v.double().view(T, heads, vdim), decays.to(DEV)[:, None, None]
    errors = [0.0, 0.0]
    for lo, hi, slot in places:
        S = first[slot].double().view(heads, dim, vdim)
        ref = torch.empty(hi - lo, heads, vdim, dtype=F64, device=DEV)
        for t in range(lo, hi):
            S = gamma * S + k[t, :, :, None] * vv[t, :, None]
            ref[t - lo] = (q[t, :, None] @ S)[:, 0]
        for i, (o, state) in enumerate(results):
            errors[i] = max(errors[i], float((o[lo:hi].double() - ref).norm() / ref.norm()),
                            float((state[slot].double().view_as(S) - S).norm() / S.norm()))
    print("chunks", errors[0], "tokens", errors[1])
    # 32-bit sums of up to 64 + 128 terms in either order: a few times 2^-24
    assert errors[0] < 2e-6 and errors[0] < 1.5 * errors[1]
    for _, state in results:                                                                # nobody else's state is touched
        assert torch.equal(state[0], first[0]) and torch.equal(state[len(lens) + 1:], first[len(lens) + 1:])
