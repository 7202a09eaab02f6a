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


@pytest.mark.parametrize("channels", [True, False])
@pytest.mark.parametrize("dim, vdim", [(64, 64), (128, 128), (64, 192)])
@pytest.mark.parametrize("lens", [[65], [64, 128], [130, 1, 17, 16, 200], [700]])
@pytest.mark.parametrize("pace", [0.02, 1.0, 30.0])          # decays next to one, ordinary ones, channels that forget at once
def test_delta_rule(dim, vdim, lens, channels, pace):
    ops, heads, kv_heads = _ops(), 4, 2
    step, places = _requests(lens)
    T, QK = sum(lens), kv_heads * dim
    g = torch.Generator().manual_seed(dim + T)
    qkv = (torch.randn(T, 2 * QK + heads * vdim, generator=g) * 0.7).bfloat16().to(DEV)
    beta = torch.randn(T, heads, generator=g).bfloat16().to(DEV)
    per = dim if channels else 1
    a, bias = torch.randn(T, heads * per, generator=g).to(DEV), (torch.randn(heads * per, generator=g) * 0.5).to(DEV)
    log = torch.log(torch.tensor([0.2, 1.0, 2.0, 0.5])).to(DEV) + torch.log(torch.tensor(pace)).to(DEV)
    first = torch.randn(len(lens) + 2, heads * dim * vdim + 4, generator=g).to(DEV)
    results = []
    for chunked in (True, False):
        state, ops.chunk_min_rows = first.clone(), 64 if chunked else 1 << 30
        o = ops.gated_delta_rule(qkv, beta, a, decay_log=log, decay_bias=bias, state=state, step=step, heads=heads,
                                 kv_heads=kv_heads, key_dim=dim, value_dim=vdim, unit_eps=1e-6, q_scale=dim ** -0.5)
        results.append((o, state))
    ops.chunk_min_rows = type(ops).chunk_min_rows
    ops.check_errors()
    x = qkv.double()
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)                     # noqa: E731
    q, k = (unit(t.view(T, kv_heads, dim)).repeat_interleave(heads // kv_heads, 1) for t in (x[:, :QK], x[:, QK:2 * QK]))
    q, v = q * dim ** -0.5, x[:, 2 * QK:].view(T, heads, vdim)
    z = (a.double() + bias.double()).view(T, heads, per)
    decay = torch.exp(-torch.exp(log.double())[:, None] * torch.nn.functional.softplus(z)).expand(T, heads, dim)
    write = torch.sigmoid(beta.double())
    errors = [0.0, 0.0]
    for lo, hi, slot in places:
        S = first[slot, :-4].double().view(heads, dim, vdim)
        ref = torch.empty(hi - lo, heads, vdim, dtype=F64, device=DEV)
        for t in range(lo, hi):
            S = decay[t, :, :, None] * S
            u = write[t, :, None] * (v[t] - (k[t, :, None] @ S)[:, 0])
            S = S + k[t, :, :, None] * u[:, None]
            ref[t - lo] = (q[t, :, None] @ S)[:, 0]
        for i, (o, state) in enumerate(results):
            errors[i] = max(errors[i], float((o[lo:hi].double() - ref).norm() / ref.norm()),
                            float((state[slot, :-4].double().view_as(S) - S).norm() / S.norm()))
    print("chunks", errors[0], "tokens", errors[1])
    # 32-bit sums of chains of up to 128 + 64 terms, where the token loop adds 4 and then by halves: a few times 2^-24 either way
    assert errors[0] < 8 * 2.0 ** -24 and errors[0] < 3 * errors[1]
    for _, state in results:
        assert torch.equal(state[0], first[0]) and torch.equal(state[len(lens) + 1:], first[len(lens) + 1:])
        assert torch.equal(state[:, -4:], first[:, -4:])
