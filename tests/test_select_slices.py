"""The sliced selection kernel at its edges — rows around a slice, every table layout for the
bitmap-decided and the later probes, keys outside the tables, unaligned columns, segment
sizes on both sides of a slice, full lists — against the oracle's selection."""
import ctypes as C

import numpy as np
import pytest
import torch

from mordred_b200 import _lib as L
from mordred_b200 import ssb
from oracle import oracle as O

pytestmark = pytest.mark.gpu
BETWEEN, EQ, EQ2 = L.MB_FILTER_BETWEEN, L.MB_FILTER_EQ, L.MB_FILTER_EQ_OR_EQ


def _table(rng, layout, slots, kmin, share):
    """A hash table whose slots are filled at random (also the wrapped one), on both sides."""
    keys = np.arange(kmin + 1, kmin + slots + 1, dtype=np.int32)
    flt = (rng.random(slots) < share).astype(np.int32)
    val = None if layout == L.MB_HT_KEY else rng.integers(0, 50, slots).astype(np.int32)
    ht = np.zeros(slots * (1 if layout == L.MB_HT_KEY else 2), np.int32)
    O.build_ht(flt, EQ, 1, 0, keys, val, ht, slots, kmin, layout)
    return ht


def _dev(a, shift=0):
    d = torch.empty(len(a) + shift, dtype=torch.int32, device="cuda")
    d[shift:] = torch.from_numpy(a).cuda()
    return d[shift:]


def _check(n, filters, probes, seed, shift=0, wild=0.0, capacity=None, segment=None):
    rng = np.random.default_rng(seed)
    hf, hp, df, dp, keep = [], [], [], [], []
    extra_h, extra_d = {}, {}
    nseg = 0
    if segment:
        S, order = segment
        nseg = max(order) + 1
        extra_h = dict(segment_group=np.array(order, np.int16), segment_size=S)
    rows = nseg * segment[0] if segment else n
    cols = []
    for mode, c1, c2 in filters:
        cols.append(rng.integers(0, 20, rows).astype(np.int32))
        hf.append(dict(col=cols[-1], mode=mode, c1=c1, c2=c2))
    for layout, slots, kmin, share in probes:
        ht = _table(rng, layout, slots, kmin, share)
        key = rng.integers(kmin + 1, kmin + slots + 1, rows).astype(np.int32)
        if wild:
            odd = rng.random(rows) < wild
            key[odd] = rng.integers(kmin - 3 * slots, kmin + 9 * slots, int(odd.sum())).astype(np.int32)
        cols.append(key)
        hp.append(dict(fkey=key, ht=ht, num_slots=slots, key_min=kmin, layout=layout))
    if segment:
        perm = rng.permutation(nseg * len(cols)).reshape(len(cols), nseg)
        pool = np.zeros(nseg * len(cols) * S, np.int32)
        for c, col in enumerate(cols):
            for g in range(nseg):
                pool[perm[c, g] * S: (perm[c, g] + 1) * S] = col[g * S: (g + 1) * S]
        dcols = [_dev(perm[c].astype(np.int32)) for c in range(len(cols))]
        keep = [_dev(pool), torch.tensor(order, dtype=torch.int16, device="cuda")]
        extra_d = dict(gpu_cache=keep[0], segment_group=keep[1], segment_size=S)
    else:
        dcols = [_dev(c, shift) for c in cols]
    for d, f in zip(dcols, hf):
        df.append(dict(f, col=d))
    for d, p in zip(dcols[len(hf):], hp):
        dp.append(dict(p, fkey=d, ht=_dev(p["ht"], 2 if shift else 0)))  # 8-byte aligned only when shifted
    a = ssb.star_args(num_rows=n, filters=df, probes=dp, **extra_d)
    cap = n if capacity is None else capacity
    lo = torch.full((max(cap, 1) + 1,), -7, dtype=torch.int32, device="cuda")
    dims = [torch.full((max(cap, 1),), -7, dtype=torch.int32, device="cuda") for _ in probes]
    total = torch.zeros(1, dtype=torch.int32, device="cuda")
    L.device_status(0)
    L.call("mb_star_select", C.byref(a), None, 0, lo.data_ptr(), (C.c_void_p * 4)(*[d.data_ptr() for d in dims]), cap,
           total.data_ptr(), ssb._stream())
    found, status = int(total.item()), L.device_status(0)
    olo, odims, k, ost = O.select(n, filters=hf, probes=hp, **extra_h)
    assert found == k and lo[-1].item() == -7
    got = lo[:min(k, cap)].cpu().numpy()
    if cap < k:
        assert status == ost | L.MB_STATUS_OVERFLOW
        assert len(np.unique(got)) == cap and np.isin(got, olo).all()
        return
    assert status == ost
    o, oo = np.argsort(got), np.argsort(olo)
    assert np.array_equal(got[o], olo[oo])
    for d, od in zip(dims, odims):
        assert np.array_equal(d[:k].cpu().numpy()[o], od[oo])


LAYOUTS = [L.MB_HT_KEY, L.MB_HT_KEY_VAL, L.MB_HT_VAL_OFF]


@pytest.mark.parametrize("n", [1, 31, 511, 512, 513, 4 * 512 * 148 - 1, 16 * 512 * 148 + 700])
@pytest.mark.parametrize("shift", [0, 1])
def test_rows_around_a_slice(n, shift):
    _check(n, [(BETWEEN, 3, 16)], [(LAYOUTS[2], 100, 0, 0.5), (LAYOUTS[1], 5_000, 0, 0.4)], n + shift, shift)


@pytest.mark.parametrize("first", LAYOUTS)
@pytest.mark.parametrize("second", [None, *LAYOUTS])
@pytest.mark.parametrize("filters", [[], [(EQ, 4, 0)], [(EQ2, 4, 9), (BETWEEN, 2, 17)],
                                     [(BETWEEN, 1, 18), (BETWEEN, 9, 3), (EQ, 1, 0)],
                                     [(BETWEEN, 1, 18), (BETWEEN, 0, 19), (BETWEEN, 2, 19)]])
def test_layouts_and_filters(first, second, filters):
    probes = [(first, 3_001, 0, 0.3)] + ([(second, 70_001, 5, 0.6), (second, 63, -7, 0.9)] if second is not None else [])
    _check(40_007, filters, probes, 7, wild=0.01)


@pytest.mark.parametrize("slots", [32, 33, 64, 65_536, 65_537])
def test_bitmap_sizes(slots):
    """Tables up to 65,536 slots are decided by the bitmap, larger ones by their loads."""
    _check(4 * 65_537 + 11, [], [(L.MB_HT_VAL_OFF, slots, 19, 0.2), (L.MB_HT_KEY, 1_000, 0, 0.5)], slots, wild=0.001)


@pytest.mark.parametrize("probes", [[], [(L.MB_HT_KEY, 65_537, 0, 0.3)], [(L.MB_HT_VAL_OFF, 2_000, 0, 0.5)] * 4])
@pytest.mark.parametrize("filters", [[], [(BETWEEN, 0, 9)]])
def test_probe_counts(filters, probes):
    _check(30_000, filters, probes, 3)


@pytest.mark.parametrize("size,order", [(256, [3, 0, 5, 1]), (512, [2, 0, 1]), (4096, [6, 1, 0, 4, 3])])
def test_segments(size, order):
    n = len(order) * size
    _check(n, [(BETWEEN, 2, 15)], [(L.MB_HT_VAL_OFF, 200, 0, 0.5), (L.MB_HT_KEY_VAL, 900, 0, 0.7)], size,
           segment=(size, order))


def test_full_list():
    _check(200_001, [], [(L.MB_HT_VAL_OFF, 500, 0, 0.9)], 9, capacity=1_000)


# one filter and two probes, the first decided by its bitmap: 23 warps an SM
@pytest.mark.parametrize("rows,slices", [(64, 23), (128, 23), (256, 23), (512, 23), (512, 60)])
@pytest.mark.parametrize("more", [-1, 0, 1, 129])
def test_slice_sizes(rows, slices, more):
    """Calls around the most rows that slices of a size take, and of more than a slice a warp."""
    _check(rows * slices * 148 + more, [(BETWEEN, 3, 16)],
           [(LAYOUTS[2], 100, 0, 0.5), (LAYOUTS[1], 5_000, 0, 0.4)], rows + more)


@pytest.mark.parametrize("first", LAYOUTS)
@pytest.mark.parametrize("second", [None, *LAYOUTS])
@pytest.mark.parametrize("filters", [[], [(BETWEEN, 1, 18), (BETWEEN, 0, 19), (BETWEEN, 2, 19)]])
def test_layouts_decided_by_a_bitmap(first, second, filters):
    """The first table's bitmap from 32 rows a slot on, the second's table read."""
    probes = [(first, 3_001, 0, 0.3)] + ([(second, 70_001, 5, 0.6), (second, 63, -7, 0.9)] if second is not None else [])
    for n in (32 * 3_001 - 1, 32 * 3_001, 700_003):
        _check(n, filters, probes, 7, wild=0.01)


@pytest.mark.parametrize("slots", [33, 65_535, 65_536, 65_537])
@pytest.mark.parametrize("layout", LAYOUTS)
def test_largest_bitmaps(slots, layout):
    _check(32 * 65_537 + 11, [], [(layout, slots, 19, 0.2), (L.MB_HT_KEY, 1_000, 0, 0.5)], slots, wild=0.001)


@pytest.mark.parametrize("share", [0.0, 0.002, 1.0])
def test_rows_dropped_before_the_last_probe(share):
    """Rounds of which no row, hardly a row and every row goes on to the second and third probe."""
    _check(300_007, [], [(L.MB_HT_VAL_OFF, 66_000, 0, share), (L.MB_HT_KEY, 500, 0, 0.5), (L.MB_HT_KEY_VAL, 66_000, 0, 0.9)],
           5, wild=0.001)


@pytest.mark.parametrize("size,order", [(512, [5, 2, 0, 1]), (1 << 16, [6, 1, 0, 4, 3])])
def test_segments_with_a_bitmap(size, order):
    _check(len(order) * size - 77, [(BETWEEN, 2, 15)], [(L.MB_HT_VAL_OFF, 60, 0, 0.5), (L.MB_HT_KEY_VAL, 900, 0, 0.7)],
           size, segment=(size, order))
