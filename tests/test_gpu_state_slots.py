"""The one-launch copy of state slots (``copy_state_slots``) against indexing, and the cache manager through it."""
import random

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    from pih_b200.kernels import get_ops
    return get_ops(torch.device("cuda:0"))


# a row of one word, of an odd number of words, a piece of 16 KB to the byte, one word beyond it, several pieces; more
# tensors than one launch takes, and more pairs
@pytest.mark.parametrize("widths, pairs", [([1], 1), ([1, 3, 4096, 4097], 5), ([12289, 64, 7], 3), ([8] * 17, 2), ([5, 4], 129)])
def test_rows_move_between_tensors(ops, widths, pairs):
    g = torch.Generator("cuda").manual_seed(3)
    src = [torch.randint(-2 ** 31, 2 ** 31 - 1, (pairs + 2, n), device="cuda", dtype=torch.int32, generator=g) for n in widths]
    dst = [torch.randint(-2 ** 31, 2 ** 31 - 1, (pairs + 3, n), device="cuda", dtype=torch.int32, generator=g) for n in widths]
    rnd = random.Random(4)
    to, of = rnd.sample(range(pairs + 3), pairs), [rnd.randrange(pairs + 2) for _ in range(pairs)]
    expected = [d.clone() for d in dst]
    for e, s in zip(expected, src):
        e[to] = s[of]
    ops.copy_state_slots(list(zip(to, of)), list(zip(dst, src)))
    for d, e in zip(dst, expected):
        assert torch.equal(d, e)
    ops.copy_state_slots([(to[0], 0)], [(d, None) for d in dst])
    for d, e in zip(dst, expected):
        e[to[0]] = 0
        assert torch.equal(d, e)


def test_a_step_of_several_requests_goes_back_together(ops):
    from pih_b200.cache import CacheManager
    from pih_b200.parts.registry import PagedKVNeed, PagedStateNeed, StateNeed
    needs = [StateNeed((5,), torch.float32), PagedStateNeed(PagedKVNeed(1, 8, None), StateNeed((2, 3), torch.float32)),
             StateNeed((1,), torch.int32)]
    m = CacheManager(needs, [None] * 3, page_size=4, num_pages=16, max_requests=4, device=torch.device("cuda:0"),
                     dtype=torch.bfloat16)
    m.slot_copier = ops.copy_state_slots
    for t in m.state_tensors.values():
        t.fill_(9)
    slots = [m.add_request(r).slot for r in "abc"]
    assert all(int(t[s].abs().sum()) == 0 for t in m.state_tensors.values() for s in slots)
    for t in m.state_tensors.values():
        t[slots] = torch.arange(1, 4, device="cuda").view((3,) + (1,) * (t.dim() - 1)).to(t.dtype)
    before = [t.clone() for t in m.state_tensors.values()]
    for rids in ("abc", "ca"):                              # two queued steps, the second of two of the requests
        for r in rids:
            m.append(r, 1, snapshot=False)
        m.snapshot_states(list(rids), torch.tensor([m.requests[r].slot for r in rids], dtype=torch.int32, device="cuda"))
        for r in rids:
            for t in m.state_tensors.values():
                t[m.requests[r].slot] += 10
            m.commit(r, confirmed=False)
    after = [t.clone() for t in m.state_tensors.values()]
    m.append("b", 2)                                        # its own copy, one request's
    for t in m.state_tensors.values():
        t[m.requests["b"].slot] += 100
    m.rollback("b")
    assert all(torch.equal(t, a) for t, a in zip(m.state_tensors.values(), after))
    m.rollback_all("abc", unconfirmed=True)
    assert all(torch.equal(t, b) for t, b in zip(m.state_tensors.values(), before))
    assert all(m.requests[r].num_tokens == 0 for r in "abc")
