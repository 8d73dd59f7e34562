"""The group keys the offset-list kernel stores: payloads of tables and passed-through values in
every order, weighed so that every tuple of keys has a group of its own, equal the oracle's word
for word — a payload of another probe, or in another slot, cannot pass."""
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


@pytest.mark.parametrize("layouts,res_layout", [
    ([VO], L.MB_RES_ENGINE6), ([PASS], L.MB_RES_ENGINE6), ([PASS, VO], L.MB_RES_CRYSTAL4),
    ([KV, PASS], L.MB_RES_CRYSTAL4), ([PASS, VO, KV], L.MB_RES_ENGINE6), ([VO, PASS, KV], L.MB_RES_ENGINE6),
    ([KV, VO, PASS, PASS], L.MB_RES_ENGINE6), ([KEY, PASS, PASS, VO], L.MB_RES_ENGINE6),
    ([KV, VO, KV, VO], L.MB_RES_ENGINE6), ([PASS, PASS, VO, KV], L.MB_RES_ENGINE6)])
@pytest.mark.parametrize("n", [300, 20_011])
@pytest.mark.parametrize("group_mode", [0, 2])
def test_stored_keys(layouts, res_layout, n, group_mode):
    rng = np.random.default_rng(n + len(layouts))
    m, radix = 3 * n, 9
    listed = rng.permutation(m)[:n].astype(np.int32)
    total = radix ** len(layouts)
    probes = []
    for j, layout in enumerate(layouts):
        slots = 300 + 17 * j
        common = dict(layout=layout, min_val=1 + j, unique_val=radix ** j, res_slot=(j + 1) % len(layouts))
        # payloads of probe j: 1 + j .. 9 + j, so that a value tells its probe apart too (KEY: 0)
        if layout == PASS:
            probes.append(dict(common, fkey=rng.integers(0, slots, n).astype(np.int32),
                               ht=rng.integers(1 + j, 10 + j, slots).astype(np.int32), num_slots=slots))
            continue
        if layout == KEY:
            common["min_val"] = 0
        keys = np.arange(1, slots + 1, dtype=np.int32)
        val = None if layout == KEY else rng.integers(1 + j, 10 + j, slots).astype(np.int32)
        ht = np.zeros(slots * (1 if layout == KEY else 2), np.int32)
        O.build_ht((rng.random(slots) < 0.7).astype(np.int32), L.MB_FILTER_EQ, 1, 0, keys, val, ht, slots, 0, layout)
        probes.append(dict(common, fkey=rng.integers(1, slots + 1, m).astype(np.int32), ht=ht, num_slots=slots))
    aggr = [rng.integers(-10**9, 10**9, m).astype(np.int32) for _ in range(2)]
    words = 3 if res_layout == L.MB_RES_ENGINE6 else 2
    kw = dict(agg_op=L.MB_AGG_SUB, total_val=total, res_layout=res_layout)
    exp = np.zeros(words * total, np.int64)
    ost = O.star(n, filters=[], probes=probes, aggr=aggr, res=exp, rows=listed, **kw)
    res = torch.zeros(words * total, dtype=torch.int64, device="cuda")
    L.device_status(0)
    ssb.star_query(ssb.star_args(num_rows=n, filters=[], probes=[dict(p, fkey=_dev(p["fkey"]), ht=_dev(p["ht"])) for p in probes],
                                 aggr=[_dev(a) for a in aggr], res=res, rows=_dev(listed), group_mode=group_mode, **kw))
    torch.cuda.synchronize()
    assert L.device_status(0) == ost == 0
    assert np.count_nonzero(exp) > 0 and np.array_equal(res.cpu().numpy(), exp)
