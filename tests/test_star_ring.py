"""The default form of star queries with probes at its edges — rows around a slice and a ring,
every table layout for the bitmap-decided, the first and the later probes, settled payloads,
keys outside the tables, counts, result layouts and groups in shared memory and L2, segment
lists, columns that are not 16-byte aligned — against the oracle."""
import itertools

import numpy as np
import pytest
import torch

from mordred_b200 import _lib as L
from mordred_b200 import ssb
from oracle import oracle as O

pytestmark = pytest.mark.gpu
KEY, KV, VO = L.MB_HT_KEY, L.MB_HT_KEY_VAL, L.MB_HT_VAL_OFF
BETWEEN, EQ, EQ2 = L.MB_FILTER_BETWEEN, L.MB_FILTER_EQ, L.MB_FILTER_EQ_OR_EQ


def _dev(a, shift=0):
    d = torch.empty(len(a) + shift, dtype=torch.int32, device="cuda")
    d[shift:] = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return d[shift:]


def _check(n, probes, seed, filters=(), agg=L.MB_AGG_SUB, res_layout=L.MB_RES_DENSE, total=175, wild=0.0, shift=0,
           count_after=-1, segment=None, group_mode=0, presence=False):
    """probes: (layout, slots, key_min, share of slots filled, group multiplier, result slot)."""
    rng = np.random.default_rng(seed)
    S, order = segment if segment else (0, [])
    m = (max(order) + 1) * S if segment else n
    cols, hf, hp, bits = [], [], [], []
    for mode, c1, c2 in filters:
        cols.append(rng.integers(0, 20, m).astype(np.int32))
        hf.append(dict(col=cols[-1], mode=mode, c1=c1, c2=c2))
    for layout, slots, kmin, share, mul, slot in probes:
        keys = np.arange(kmin + 1, kmin + slots + 1, dtype=np.int32)
        val = None if layout == KEY else rng.integers(0, 7, slots).astype(np.int32)
        ht = np.zeros(slots * (1 if layout == KEY else 2), np.int32)
        O.build_ht((rng.random(slots) < share).astype(np.int32), EQ, 1, 0, keys, val, ht, slots, kmin, layout)
        k = rng.integers(kmin + 1, kmin + slots + 1, m).astype(np.int32)
        if wild:
            odd = rng.random(m) < wild
            k[odd] = rng.integers(kmin - 3 * slots, kmin + 9 * slots, int(odd.sum())).astype(np.int32)
        cols.append(k)
        hp.append(dict(fkey=k, ht=ht, num_slots=slots, key_min=kmin, layout=layout, min_val=1, unique_val=mul,
                       res_slot=slot))
        on = ht != 0 if layout == KEY else ht.reshape(-1, 2).any(1)
        packed = np.zeros((slots + 31) // 32 * 32, np.uint8)
        packed[:slots] = on
        bits.append(np.packbits(packed, bitorder="little").view(np.int32))
    cols += [rng.integers(-10**9, 10**9, m).astype(np.int32) for _ in range(2)]
    two = agg in (L.MB_AGG_SUB, L.MB_AGG_MUL)
    extra_h, extra_d, keep = {}, {}, []
    if segment:
        perm = rng.permutation((max(order) + 1) * len(cols)).reshape(len(cols), -1)
        pool = np.zeros(perm.size * S, np.int32)
        for c, col in enumerate(cols):
            for g in range(max(order) + 1):
                pool[perm[c, g] * S: (perm[c, g] + 1) * S] = col[g * S: (g + 1) * S]
        keep = [_dev(pool), torch.tensor(order, dtype=torch.int16, device="cuda")]
        dcols = [_dev(perm[c].astype(np.int32)) for c in range(len(cols))]
        extra_h = dict(segment_group=np.array(order, np.int16), segment_size=S)
        extra_d = dict(gpu_cache=keep[0], segment_group=keep[1], segment_size=S)
    else:
        dcols = [_dev(c, shift) for c in cols]
    size = {L.MB_RES_SCALAR: 1, L.MB_RES_ENGINE6: 3 * total, L.MB_RES_CRYSTAL4: 2 * total, L.MB_RES_DENSE: total}[res_layout]
    kw = dict(agg_op=agg, total_val=total, group_bias=3, res_layout=res_layout, count_after=count_after)
    exp, ecnt = np.zeros(size, np.int64), np.zeros(1, np.uint64)
    ost = O.star(n, filters=hf, probes=hp, aggr=cols[-2:][: 1 + two], res=exp, count=ecnt, **kw, **extra_h)
    res = torch.zeros(size, dtype=torch.int64, device="cuda")
    cnt = torch.zeros(1, dtype=torch.int64, device="cuda")
    df = [dict(f, col=d) for f, d in zip(hf, dcols)]
    dp = [dict(p, fkey=d, ht=_dev(p["ht"], 2 if shift else 0), presence=_dev(b) if presence else None)
          for p, d, b in zip(hp, dcols[len(hf):], bits)]
    L.device_status(0)
    ssb.star_query(ssb.star_args(num_rows=n, filters=df, probes=dp, aggr=dcols[-2:][: 1 + two], res=res, count=cnt,
                                 group_mode=group_mode, **kw, **extra_d))
    torch.cuda.synchronize()
    assert L.device_status(0) == ost
    assert int(cnt.item()) == int(ecnt[0])
    got = res.cpu().numpy()
    if res_layout in (L.MB_RES_SCALAR, L.MB_RES_DENSE):
        assert np.array_equal(got, exp)
        return
    stride = 6 if res_layout == L.MB_RES_ENGINE6 else 4
    assert np.array_equal(got.view(np.int32).reshape(total, stride), exp.view(np.int32).reshape(total, stride))


# groups 7 x 25: date-like and nation-like payloads of 0..6 with multipliers that keep them apart
S_ = (KEY, 3_000, 0, 0.3, 0, -1)
C_ = (KV, 70_000, 0, 0.4, 7, 1)
P_ = (KEY, 70_000, 5, 0.5, 0, -1)
D_ = (KV, 61, -9, 0.9, 1, 0)


@pytest.mark.parametrize("n", [1, 63, 255, 256, 257, 1_000, 4 * 256 * 148 + 17, 70 * 256 * 148 + 5])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows_around_a_slice(n, shift):
    _check(n, [S_, C_, P_, D_], n, shift=shift, res_layout=L.MB_RES_CRYSTAL4, total=175)


@pytest.mark.parametrize("first", [KEY, KV, VO])
@pytest.mark.parametrize("lead", [KEY, KV, VO])
@pytest.mark.parametrize("later", [KEY, KV, VO])
@pytest.mark.parametrize("read_first", [0, 1])
def test_layouts(first, lead, later, read_first):
    """A small table decided by its bitmap (payload read or not), a large one, two later ones."""
    _check(150_001, [(first, 1_025, 0, 0.4, 49 * read_first, 2 if read_first else -1), (lead, 66_000, 3, 0.5, 7, 1),
                     (later, 66_000, 0, 0.7, 1, 0), (KEY, 66_001, 0, 0.8, 0, -1)], 5, wild=0.002,
           res_layout=L.MB_RES_ENGINE6, total=400)


@pytest.mark.parametrize("probes", [[S_], [C_], [D_, S_], [(VO, 40, 0, 1.0, 1, 0)] * 4, [C_, D_, S_], [S_, D_]])
@pytest.mark.parametrize("filters", [[], [(BETWEEN, 2, 15)], [(EQ2, 3, 8), (BETWEEN, 0, 12)],
                                     [(EQ, 4, 0), (BETWEEN, 9, 2), (BETWEEN, 0, 19)]])
@pytest.mark.parametrize("layout", [L.MB_RES_SCALAR, L.MB_RES_DENSE])
def test_probe_and_filter_counts(probes, filters, layout):
    if layout == L.MB_RES_SCALAR:
        probes = [(*p[:4], 0, -1) for p in probes]
    for after in (-1, 0, len(filters)):
        _check(90_001, probes, 11, filters, res_layout=layout, count_after=after, wild=0.003)


@pytest.mark.parametrize("order", list(itertools.permutations(range(4))))
def test_settled_probes_wherever_they_stand(order):
    """Two probes settled by their bitmap (one with a group term), one read for its payload, one
    without a bitmap, in every order."""
    probes = [(KEY, 3_000, 0, 0.6, 3, -1), D_, (VO, 500, 0, 0.7, 0, -1), C_]
    _check(100_003, [probes[i] for i in order], 3, wild=0.002, res_layout=L.MB_RES_ENGINE6, total=175)


@pytest.mark.parametrize("total,group_mode", [(175, 0), (175, 2), (2_048, 0), (2_049, 0), (9_000, 0)])
@pytest.mark.parametrize("agg", [L.MB_AGG_SUM, L.MB_AGG_SUB, L.MB_AGG_MUL])
def test_groups_and_aggregates(total, group_mode, agg):
    _check(120_003, [S_, C_, D_], total, agg=agg, total=total, group_mode=group_mode)


@pytest.mark.parametrize("share", [0.0, 0.02, 1.0])
def test_survivor_shares(share):
    """No row, a few rows, and every row of a slice reaches the ring."""
    _check(100_007, [(KEY, 900, 0, share, 0, -1), (KV, 66_000, 0, share, 7, 1), (VO, 66_000, 0, 1.0, 1, 0)], 2)


@pytest.mark.parametrize("slots", [31, 32, 33, 65_536, 262_144, 262_145])
@pytest.mark.parametrize("layout", [KEY, KV])
@pytest.mark.parametrize("presence", [False, True])
def test_bitmap_sizes(slots, layout, presence):
    _check(1_100_003, [(layout, slots, 2, 0.3, 0, -1), (KV, 500, 0, 0.6, 1, 0)], slots, wild=0.001, presence=presence)


@pytest.mark.parametrize("slots,n", [(20_000, 80_000), (20_000, 79_999), (20_001, 640_032), (20_001, 640_031),
                                     (65_536, 2_097_152), (65_536, 2_097_151)])
@pytest.mark.parametrize("layout", [KV, VO])
def test_rows_from_which_a_bitmap_is_derived(slots, n, layout):
    """Tables of 8-byte slots: 4 rows a slot, above 20,000 slots 32."""
    _check(n, [(layout, slots, 2, 0.3, 7, 1), (KEY, 500, 0, 0.6, 0, -1)], slots, wild=0.001, res_layout=L.MB_RES_ENGINE6)


@pytest.mark.parametrize("size,order", [(2048, [3, 0, 5, 1]), (4096, [6, 1, 0, 4, 3])])
def test_segments(size, order):
    _check(len(order) * size - 5, [S_, C_, P_, D_], size, [(BETWEEN, 1, 18)], segment=(size, order))
