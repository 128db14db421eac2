"""The cache's bookkeeping: no slot or page lost, held twice or freed twice; groups; windows."""
import random

import pytest
import torch

import bitnet_c_b200  # noqa: F401
from bitnet_c_b200.cache import PAGE, Cache, CacheError, CacheFull, PagePool, SlotTable, pages_for
from bitnet_c_b200.parts import KvRequest, StateRequest


def make(kv, cache_of=None, states=None, max_tokens=640, max_positions=512, max_seqs=4):
    n = len(kv)
    return Cache(kv, cache_of or [None] * n, states or [None] * n, max_tokens, max_positions, torch.bfloat16,
                 None, max_seqs=max_seqs, allocate=False)


def test_page_pool_never_loses_or_doubles():
    p = PagePool(10)
    a = p.alloc(4)
    b = p.alloc(6)
    assert sorted(a + b) == list(range(10)) and p.n_free == 0
    with pytest.raises(CacheFull):
        p.alloc(1)
    p.free(a)
    with pytest.raises(CacheError, match="freed twice"):
        p.free([a[0]])
    with pytest.raises(CacheError, match="does not exist"):
        p.free([99])
    p.check()
    assert sorted(p.alloc(4)) == sorted(a)


def test_slot_table():
    s = SlotTable(3)
    a, b, c = s.open(), s.open(), s.open()
    assert {a, b, c} == {0, 1, 2}
    with pytest.raises(CacheFull):
        s.open()
    s.close(b)
    with pytest.raises(CacheError, match="not open"):
        s.close(b)
    with pytest.raises(CacheError):
        s.length(b)
    assert s.open() == b  # given back and used again
    s.check()


def test_reserve_advance_close_cycle_many_times():
    req = KvRequest(2, 16)
    c = make([req, req, req])
    assert len(c.groups) == 1 and c.groups[0].entries == [0, 1, 2]
    rng = random.Random(0)
    live = {}
    for _ in range(500):
        if live and (rng.random() < 0.3 or c.slots.n_free == 0):
            slot = rng.choice(list(live))
            c.close(slot)
            del live[slot]
        elif rng.random() < 0.5 or not live:
            live[c.open()] = 0
        else:
            slot = rng.choice(list(live))
            n = rng.choice([1, 1, 1, 7, 64, 100])
            try:
                c.reserve(slot, n)
                c.advance(slot, n)
                live[slot] += n
            except CacheFull:
                pass
        c.check()
        for slot, n in live.items():
            assert c.length(slot) == n
            assert len(c.groups[0].held.get(slot, {})) == pages_for(n)
    for slot in list(live):
        c.close(slot)
    c.check()
    assert c.groups[0].pool.n_free == c.groups[0].pool.n_pages and c.slots.n_free == 4


def test_failed_reserve_changes_nothing():
    c = make([KvRequest(1, 16)], max_tokens=128, max_positions=4096)
    a, b = c.open(), c.open()
    c.reserve(a, 64)
    c.advance(a, 64)
    c.reserve(b, 10)
    c.advance(b, 10)
    with pytest.raises(CacheFull):
        c.reserve(a, 1)  # would need a third page
    assert c.length(a) == 64 and len(c.groups[0].held[a]) == 1
    c.check()
    small = make([KvRequest(1, 16)], max_positions=100)
    with pytest.raises(CacheFull, match="exceed the context"):
        small.reserve(small.open(), 101)
    small.check()


def test_groups_have_storage_of_their_own_and_readers_share_a_plane():
    full, win = KvRequest(2, 16), KvRequest(2, 16, window=70)
    c = make([full, win, None, full, win], cache_of=[None, None, None, 0, None],
             states=[None, None, StateRequest((3, 5)), None, None])
    assert [g.request for g in c.groups] == [full, win]
    assert c.groups[0].entries == [0] and c.groups[1].entries == [1, 4]
    assert c._reader == {3: 0}
    slot = c.open()
    for _ in range(5):
        c.reserve(slot, 64)
        c.advance(slot, 64)
        c.check()
    # 320 tokens: the full group holds 5 pages; the window group only pages that still hold one
    # of the last 70 keys (positions 251..319 -> pages 3 and 4)
    assert sorted(c.groups[0].held[slot]) == [0, 1, 2, 3, 4]
    assert sorted(c.groups[1].held[slot]) == [3, 4]
    c.close(slot)
    c.check()
    with pytest.raises(CacheError, match="which has none"):
        make([None, full], cache_of=[None, 0])
    with pytest.raises(CacheError, match="cannot read"):
        make([full, KvRequest(4, 16)], cache_of=[None, 0])


def test_sizes_round_up_to_pages():
    c = make([KvRequest(1, 16)], max_tokens=100)
    assert c.max_tokens == 128 and c.groups[0].pool.n_pages == 2 and PAGE == 64
    assert c.tokens_free() == 128


@pytest.mark.parametrize("stateful", [False, True])
def test_the_kernel_that_zeroes_states_is_built_with_the_model(stateful):
    """Opening a sequence of a model with states launches it: it must not be the first request that has it compiled."""
    import rudolix_cases
    import tiny_configs
    from bitnet_c_b200.config import architecture_of
    cfg = rudolix_cases.CASE_A if stateful else tiny_configs.TINY_A
    arch = architecture_of(cfg)
    model = bitnet_c_b200.Model(arch.to_spec(arch.read_config(cfg)), dtype="float32", device=None)
    assert ("cache_rows" in model.kernel_families()) == stateful


def test_own_planes_are_what_the_views_show_or_none():
    """Addresses for a launch over several entries: those of the views, and none at all unless every entry is as it is asked for."""
    kv, cpu = KvRequest(2, 16), torch.device("cpu")

    def cache(requests, cache_of=None, dtype=torch.bfloat16):
        return Cache(requests, cache_of or [None] * len(requests), [None] * len(requests), 640, 512, dtype, cpu, max_seqs=4)

    mixed = [kv, KvRequest(2, 16, window=128), kv]  # two groups
    c = cache(mixed)
    got = c.own_planes(3, 2, 16, torch.bfloat16, cpu)
    for i, (k, v, table, row, pages) in enumerate(got):
        view = c.view(i)
        assert (k, v, table) == (view.k.data_ptr(), view.v.data_ptr(), view.page_table.data_ptr())
        assert (row, pages) == (view.page_table.shape[1], view.k.shape[0])
    assert len({k for k, *_ in got}) == 3
    assert c.own_planes(4, 2, 16, torch.bfloat16, cpu) is None  # more entries than it has
    assert c.own_planes(3, 1, 16, torch.bfloat16, cpu) is None and c.own_planes(3, 2, 32, torch.bfloat16, cpu) is None
    assert c.own_planes(3, 2, 16, torch.float32, cpu) is None and c.own_planes(3, 2, 16, torch.bfloat16, torch.device("meta")) is None
    assert cache(mixed, dtype=torch.float32).own_planes(3, 2, 16, torch.bfloat16, cpu) is None
    assert cache([kv, kv], [None, 0]).own_planes(2, 2, 16, torch.bfloat16, cpu) is None  # an entry that reads another's
    for other in (KvRequest(4, 16), KvRequest(2, 32), KvRequest(2, 16, v_head_dim=8), KvRequest(2, 16, values_in_keys=True), None):
        assert cache([kv, other]).own_planes(2, 2, 16, torch.bfloat16, cpu) is None
        assert len(cache([kv, other]).own_planes(1, 2, 16, torch.bfloat16, cpu)) == 1
