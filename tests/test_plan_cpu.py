"""Host-side planner of balanced launches (miniattn_plan_fwd): pure arithmetic, no device.

A plan cuts the K/V tile range of some work items into pieces for separate CTAs.  Whatever the
shape, the pieces of an item must tile its range exactly once, slots must be unique, and the plan
must only be used when its predicted makespan beats the plain launch.
"""
import collections

import pytest

from miniattn.ops import plan_info

SMS = 148


def item_tiles(item, B, Hq, Nq, Nk, causal, q_pos0=0, k_pos0=0, group=None):
    """K/V tiles of work item `item` (pair of 128-row Q tiles): heads walked in groups of `group`
    (all B*Hq at once by default), inside a group latest rows first, heads fastest."""
    n_pairs = ((Nq + 127) // 128 + 1) // 2
    group = group or B * Hq
    pair = n_pairs - 1 - (item % (n_pairs * group)) // group
    q0 = pair * 256
    nt = 2 if q0 + 128 < Nq else 1
    kv_end = Nk
    if causal:
        last_row = min(q0 + nt * 128 - 1, Nq - 1)
        kv_end = max(0, min(Nk, q_pos0 + last_row - k_pos0 + 1))
    return (kv_end + 127) // 128


CASES = [
    # B, Hq, Nq, Nk, D, causal, q_pos0, k_pos0
    (2, 8, 8192, 8192, 128, False, 0, 0),
    (2, 8, 4096, 4096, 128, False, 0, 0),
    (2, 8, 1024, 1024, 128, False, 0, 0),
    (1, 1, 8192, 8192, 128, False, 0, 0),
    (1, 4, 4096, 4096, 128, True, 0, 0),
    (1, 3, 1000, 5000, 64, True, 4000, 0),
    (1, 2, 900, 3000, 128, True, 0, 500),
    (3, 5, 2304, 1111, 64, False, 0, 0),
    (1, 16, 8192, 8192, 128, False, 0, 0),
]


@pytest.mark.parametrize("case", CASES)
def test_pieces_tile_every_item_once(case):
    B, Hq, Nq, Nk, D, causal, qp, kp = case
    info, pieces = plan_info(B, Hq, Nq, Nk, D, causal=causal, q_pos0=qp, k_pos0=kp, sm_count=SMS)
    n_items = (((Nq + 127) // 128 + 1) // 2) * B * Hq
    if not info.split:
        assert info.n_ctas == n_items and info.scratch_bytes == 0 and not pieces
        return
    assert info.n_ctas == info.n_whole + info.n_pieces == info.n_whole + len(pieces)
    by_item = collections.defaultdict(list)
    for item, t0, t1, part, nparts, slot in pieces:
        assert item >= info.n_whole, "an item of the whole prefix must not appear in the table"
        by_item[item].append((part, t0, t1, nparts, slot))
    assert sorted(by_item) == list(range(info.n_whole, n_items)), "every other item is in the table"
    slots = []
    cut = 0
    for item, lst in by_item.items():
        lst.sort()
        w = item_tiles(item, B, Hq, Nq, Nk, causal, qp, kp, info.head_group)
        assert [x[0] for x in lst] == list(range(len(lst)))
        assert all(x[3] == len(lst) for x in lst)
        assert lst[0][1] == 0 and lst[-1][2] == w, (item, lst, w)
        for a, b_ in zip(lst, lst[1:]):
            assert a[2] == b_[1], "pieces must be contiguous"
        if len(lst) > 1:
            cut += 1
            assert all(x[2] - x[1] >= 2 for x in lst), "no piece shorter than two K/V tiles"
            slots += [x[4] for x in lst]
            assert [x[4] for x in lst] == list(range(lst[0][4], lst[0][4] + len(lst))), "consecutive slots"
        else:
            assert lst[0][4] == -1
    assert cut == info.n_cut_items and sorted(slots) == list(range(info.n_slots))
    rows = info.n_slots * 2 * 128
    assert info.scratch_bytes == 16384 + ((rows * 8 + 255) // 256) * 256 + rows * D * 4
    assert info.est_balanced <= 0.97 * info.est_plain
    assert info.n_pieces <= 768


def test_headline_shapes_are_split_and_big_grids_are_not():
    assert plan_info(2, 8, 8192, 8192, sm_count=SMS)[0].split == 1      # 512 items: 3.46 rounds
    assert plan_info(2, 8, 4096, 4096, sm_count=SMS)[0].split == 1      # 256 items: 1.73 rounds
    assert plan_info(2, 8, 2048, 2048, sm_count=SMS)[0].split == 0      # 128 items in one round
    assert plan_info(4, 32, 4096, 4096, causal=True, sm_count=SMS)[0].split == 0   # 2048 items
    assert plan_info(1, 32, 131072, 131072, causal=True, sm_count=SMS)[0].split == 0
    info, _ = plan_info(2, 8, 8192, 8192, sm_count=SMS)
    assert info.n_whole == 444 and info.n_cut_items == 68   # three whole rounds, the rest is cut


def test_plan_is_deterministic_and_depends_on_sm_count():
    a = plan_info(2, 8, 4096, 4096, sm_count=SMS)
    b = plan_info(2, 8, 4096, 4096, sm_count=SMS)
    assert a[1] == b[1] and a[0].n_slots == b[0].n_slots
    c = plan_info(2, 8, 4096, 4096, sm_count=128)   # 256 items on 128 SMs: two full rounds
    assert c[0].split == 0


def test_empty_and_degenerate_shapes():
    assert plan_info(0, 8, 512, 512, sm_count=SMS)[0].split == 0
    assert plan_info(2, 8, 512, 0, sm_count=SMS)[0].split == 0
    info, _ = plan_info(1, 1, 128, 128, sm_count=SMS)      # one item, one K/V tile: nothing to cut
    assert info.split == 0 and info.n_ctas == 1


def test_random_shapes_keep_the_invariants():
    """Seeded sweep over shapes, masks, offsets and SM counts: whatever the planner decides, the
    pieces it hands out must tile every item exactly once."""
    import random
    rng = random.Random(7)
    n_split = 0
    for _ in range(120):
        B, Hq = rng.randint(1, 3), rng.randint(1, 12)
        Nq, Nk = rng.randint(1, 40) * rng.choice([100, 128, 256]), rng.randint(1, 60) * rng.choice([100, 128])
        D = rng.choice([64, 128])
        causal = rng.random() < 0.5
        qp = rng.choice([0, 0, max(0, Nk - Nq), rng.randint(0, 3000)]) if causal else 0
        kp = rng.choice([0, 0, rng.randint(0, 500)]) if causal else 0
        sms = rng.choice([148, 132, 64, 16])
        info, pieces = plan_info(B, Hq, Nq, Nk, D, causal=causal, q_pos0=qp, k_pos0=kp, sm_count=sms)
        n_items = (((Nq + 127) // 128 + 1) // 2) * B * Hq
        if not info.split:
            assert info.n_ctas == n_items
            continue
        n_split += 1
        cover = collections.defaultdict(list)
        for item, t0, t1, part, nparts, slot in pieces:
            assert info.n_whole <= item < n_items and 0 <= t0 <= t1
            cover[item].append((t0, t1, nparts, slot))
        assert len(cover) == n_items - info.n_whole
        for item, lst in cover.items():
            lst.sort()
            w = item_tiles(item, B, Hq, Nq, Nk, causal, qp, kp, info.head_group)
            assert lst[0][0] == 0 and lst[-1][1] == w and all(a[1] == b_[0] for a, b_ in zip(lst, lst[1:]))
            assert all(x[2] == len(lst) for x in lst)
            assert all((x[3] >= 0) == (len(lst) > 1) for x in lst)
        assert info.est_balanced <= 0.97 * info.est_plain
    assert n_split >= 20, "the sweep must exercise the cutting path"


def test_plan_entry_rejects_bad_arguments():
    import ctypes as C
    from miniattn import _lib
    p = _lib.FwdParams()
    p.B, p.Hq, p.Hkv, p.Nq, p.Nk, p.D = 1, 1, 1, 128, 128, 80
    info = _lib.PlanInfo()
    assert _lib.lib.miniattn_plan_fwd(C.byref(p), 148, C.byref(info), None, 0) == _lib.EUNSUPPORTED
    p.D = 128
    assert _lib.lib.miniattn_plan_fwd(C.byref(p), 148, None, None, 0) == _lib.EINVAL
    p.Nq = -1
    assert _lib.lib.miniattn_plan_fwd(C.byref(p), 148, C.byref(info), None, 0) == _lib.EINVAL


def _fwd_params(B, Hq, Hkv, Nq, Nk, D, causal=True):
    from miniattn import _lib
    p = _lib.FwdParams()
    p.B, p.Hq, p.Hkv, p.Nq, p.Nk, p.D, p.causal = B, Hq, Hkv, Nq, Nk, D, int(causal)
    p.q_pos0 = Nk - Nq if causal else 0
    return p


def _scratch(p, int8qk=0):
    import ctypes as C
    from miniattn import _lib
    need = _lib.lib.miniattn_fwd_scratch_bytes(C.byref(p), int8qk, SMS)
    assert need >= 0
    return need


def test_a_growing_context_is_not_planned_for_at_every_token():
    """Sizing the scratch of a decode call makes no plan of the general kernel; sizing an INT8-QK one, or a general
    call of a few hundred rows, makes one for each new count of K/V tiles.  A plan takes 0.5 to 4 ms: two thousand
    of them take seconds, and the bound is a tenth of one."""
    import time
    t0 = time.perf_counter()
    needs = {_scratch(_fwd_params(16, 32, 8, 1, 4001 + i, 128)) for i in range(2000)}
    assert max(needs) > 0 and time.perf_counter() - t0 < 0.1
    t0 = time.perf_counter()
    for i in range(2000):                       # 16 counts of tiles
        _scratch(_fwd_params(2, 8, 8, 600, 4001 + i, 64, causal=False), i % 2)
    assert time.perf_counter() - t0 < 0.5


def test_plans_of_the_same_tiles_are_the_same():
    """Key counts inside one 128-key tile visit the same tiles; across the boundary they do not."""
    a, b, c = (plan_info(1, 6, 1024, nk, 128, sm_count=SMS) for nk in (4001, 4096, 4097))
    assert a[0].split and a[1] == b[1] and a[0].scratch_bytes == b[0].scratch_bytes
    assert a[1] != c[1]
    d, e = (plan_info(b_, h, 1024, 4096, 128, sm_count=SMS) for b_, h in ((2, 3), (1, 6)))
    assert d[1] == e[1]                         # the items are the same, whatever B and H are one by one


def test_scratch_of_either_launch():
    """Decode: the pieces of the few-rows kernel.  INT8-QK: the general kernel's plan without packed heads."""
    p = _fwd_params(2, 24, 8, 777, 3333, 128)
    assert _scratch(p, 1) == plan_info(2, 24, 777, 3333, 128, causal=True, q_pos0=3333 - 777, sm_count=SMS)[0].scratch_bytes
    q = _fwd_params(1, 8, 1, 1, 8192, 128)
    assert 16384 < _scratch(q) < 16384 + 2 * 2 * SMS * 16 * (8 + 4 * 128)
    assert _scratch(q, 1) == plan_info(1, 8, 1, 8192, 128, causal=True, q_pos0=8191, sm_count=SMS)[0].scratch_bytes
    q.carry_in = 1
    assert _scratch(q) == 0


def test_more_shapes_in_rotation_than_a_handful():
    import time
    shapes = [_fwd_params(1, 12, 4, 500 + 64 * i, 3000, 128) for i in range(40)]
    t = []
    for _ in range(2):
        t0 = time.perf_counter()
        for p in shapes:
            _scratch(p)
        t.append(time.perf_counter() - t0)
    assert t[1] < t[0] / 4


def _packs(B, Hkv, G, Nq, Nk, causal, q_pos0):
    """Whether the rule packs the G heads, read off the number of work items (G = 1 or 0 pairs apart: unknown)."""
    import ctypes as C
    from miniattn import _lib
    p = _fwd_params(B, Hkv * G, Hkv, Nq, Nk, 128, causal)
    p.q_pos0, p.carry_in = q_pos0, 0
    p.B = 65535                                  # too many items to plan: n_ctas is their number
    info = _lib.PlanInfo()
    _lib.check(_lib.lib.miniattn_plan_fwd(C.byref(p), SMS, C.byref(info), None, 0), "plan")
    plain = (((Nq + 127) // 128 + 1) // 2) * Hkv * G
    tpt = 128 // G
    packed = (((Nq + tpt - 1) // tpt + 1) // 2) * Hkv
    items = info.n_ctas // 65535
    assert items in (plain, packed)
    return None if plain == packed else items == packed


def _rule(G, Nq, Nk, causal, pos):
    """The rule stated pair by pair: packed where that saves at least 1 % of the weighted K/V tiles."""
    def visits(tpt):
        n, s = -(-Nq // tpt), 0
        for t in range(0, n, 2):
            nt = 2 if t + 1 < n else 1
            end = Nk if not causal else max(0, min(Nk, pos + min((t + nt) * tpt, Nq)))
            s += (3 if nt == 2 else 2) * -(-end // 128)
        return s
    return visits(128 // G) * 100 <= visits(128) * G * 99


def test_head_packing_rule_in_closed_form():
    import random
    rng = random.Random(5)
    seen = [0, 0]
    for _ in range(3000):
        G = rng.choice([2, 3, 4, 5, 7, 8, 16, 48, 64, 128])
        Nq, Nk = (int(2 ** rng.uniform(0, 15)) for _ in range(2))
        causal = rng.random() < 0.8
        pos = rng.choice([0, Nk - Nq, rng.randrange(-Nq - 300, Nk + 300)]) if causal else 0
        got = _packs(1, 1, G, Nq, Nk, causal, pos)
        if got is not None:
            assert got == _rule(G, Nq, Nk, causal, pos), (G, Nq, Nk, causal, pos)
            seen[got] += 1
    assert min(seen) > 200


def test_head_packing_rule_takes_no_time_over_many_pairs():
    """128 heads share a KV head: a Q tile holds one token and 131072 rows have 65536 pairs.  A walk over them took
    150 us a call; the bound is a fifth of that."""
    import ctypes as C
    import time
    from miniattn import _lib
    p = _fwd_params(1, 128, 1, 131072, 131072, 128)
    info = _lib.PlanInfo()
    t0 = time.perf_counter()
    for _ in range(1000):
        _lib.lib.miniattn_plan_fwd(C.byref(p), SMS, C.byref(info), None, 0)
    assert time.perf_counter() - t0 < 0.03
