"""The offset-list kernel's rounds — tables and passed-through values in every order, filters
before them, keys and dimension rows out of range, list lengths around a thread's entries —
against the oracle's list form."""
import numpy as np
import pytest
import torch

from mordred_b200 import _lib as L
from mordred_b200 import ssb
from oracle import oracle as O

pytestmark = pytest.mark.gpu
KEY, KV, VO, PASS = L.MB_HT_KEY, L.MB_HT_KEY_VAL, L.MB_HT_VAL_OFF, L.MB_HT_PASS


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _check(n, layouts, seed, agg, res_layout, total, wild=0.0, filters=1, rows=True):
    rng = np.random.default_rng(seed)
    m = 4 * n + 100
    listed = rng.permutation(m)[:n].astype(np.int32) if rows else None
    hf, hp = [], []
    for _ in range(filters):
        hf.append(dict(col=rng.integers(0, 10, m).astype(np.int32), mode=L.MB_FILTER_BETWEEN, c1=1, c2=8))
    for j, layout in enumerate(layouts):
        slots = 300 + 17 * j
        slot = j if res_layout == L.MB_RES_ENGINE6 else (j if j < 2 and res_layout == L.MB_RES_CRYSTAL4 else -1)
        common = dict(layout=layout, min_val=j, unique_val=[1, 7, 0, 31][j], res_slot=slot)
        if layout == PASS:
            d = rng.integers(0, slots, n if rows else m).astype(np.int32)
            if wild:
                odd = rng.random(len(d)) < wild
                d[odd] = rng.integers(-5, slots + 5, int(odd.sum())).astype(np.int32)
            hp.append(dict(common, fkey=d, ht=rng.integers(0, 6, slots).astype(np.int32), num_slots=slots))
            continue
        keys = np.arange(1, slots + 1, dtype=np.int32)
        val = None if layout == KEY else rng.integers(0, 9, slots).astype(np.int32)
        ht = np.zeros(slots * (1 if layout == KEY else 2), np.int32)
        O.build_ht((rng.random(slots) < 0.6).astype(np.int32), L.MB_FILTER_EQ, 1, 0, keys, val, ht, slots, 0, layout)
        k = rng.integers(1, slots + 1, m).astype(np.int32)
        if wild:
            odd = rng.random(m) < wild
            k[odd] = rng.integers(-4 * slots, 7 * slots, int(odd.sum())).astype(np.int32)
        hp.append(dict(common, fkey=k, ht=ht, num_slots=slots))
    aggr = [rng.integers(-10**9, 10**9, m).astype(np.int32) for _ in range(2)]
    two = agg in (L.MB_AGG_SUB, L.MB_AGG_MUL)
    size = {L.MB_RES_SCALAR: 1, L.MB_RES_ENGINE6: 3 * total, L.MB_RES_CRYSTAL4: 2 * total, L.MB_RES_DENSE: total}[res_layout]
    kw = dict(agg_op=agg, total_val=total, group_bias=5, res_layout=res_layout)
    exp = np.zeros(size, np.int64)
    ecnt = np.zeros(1, np.uint64)
    ost = O.star(n, filters=hf, probes=hp, aggr=aggr[: 1 + two], res=exp, rows=listed, count=ecnt, count_after=-1, **kw)
    res = torch.zeros(size, dtype=torch.int64, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    dp = [dict(p, fkey=_dev(p["fkey"]), ht=_dev(p["ht"])) for p in hp]
    df = [dict(f, col=_dev(f["col"])) for f in hf]
    da = [_dev(a) for a in aggr[: 1 + two]]
    dl = _dev(listed) if rows else None
    L.device_status(0)
    ssb.star_query(ssb.star_args(num_rows=n, filters=df, probes=dp, aggr=da, res=res, rows=dl, count=cnt,
                                 count_after=-1, **kw))
    torch.cuda.synchronize()
    assert L.device_status(0) == ost
    assert int(cnt.item()) == int(ecnt[0])
    got = res.cpu().numpy()
    if res_layout in (L.MB_RES_SCALAR, L.MB_RES_DENSE):
        assert np.array_equal(got, exp)
        return
    stride = 6 if res_layout == L.MB_RES_ENGINE6 else 4
    g, e = (a.view(np.int32).reshape(total, stride) for a in (got, exp))
    assert np.array_equal(g[:, stride - 2:], e[:, stride - 2:])
    # several key tuples can share a group (the index wraps): keys are set in the same groups
    assert np.array_equal(g[:, : stride - 2].any(1), e[:, : stride - 2].any(1)) or total < 2_000


@pytest.mark.parametrize("layouts", [[], [VO], [PASS], [PASS, VO, VO], [VO, PASS, KV], [KEY, PASS, PASS, VO],
                                     [KV, VO, KEY, VO], [PASS, PASS], [VO, VO, VO, PASS]])
@pytest.mark.parametrize("res_layout,total", [(L.MB_RES_SCALAR, 1), (L.MB_RES_DENSE, 175), (L.MB_RES_DENSE, 9_000),
                                              (L.MB_RES_ENGINE6, 2_500)])
def test_orders_of_tables_and_passed_values(layouts, res_layout, total):
    if not layouts and res_layout == L.MB_RES_ENGINE6:
        pytest.skip("no keys to store")
    _check(20_011, layouts, len(layouts) + total, L.MB_AGG_SUB, res_layout, total, wild=0.01)


@pytest.mark.parametrize("n", [1, 255, 256, 257, 511, 513, 2 * 256 * 3 * 148 + 5])
@pytest.mark.parametrize("agg", [L.MB_AGG_SUM, L.MB_AGG_SUB, L.MB_AGG_MUL, L.MB_AGG_MUL_PAYLOAD])
def test_list_lengths_and_aggregates(n, agg):
    _check(n, [KV, PASS], n, agg, L.MB_RES_DENSE, 300, filters=n % 4)


def test_passed_values_without_a_list():
    _check(30_001, [PASS, VO], 4, L.MB_AGG_MUL, L.MB_RES_CRYSTAL4, 2_100, rows=False)
