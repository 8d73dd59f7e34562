"""Clearing and building a query's tables together (mb_build_tables) against the oracle's
builds, at row counts around a thread's and a block's rows, for aligned and unaligned columns,
dirty tables, presence bitmaps and a cleared result range; and the single builds of the same
kernel."""
import numpy as np
import pytest
import torch

from mordred_b200 import _lib as L
from mordred_b200 import ssb
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _dev(a, shift=0):
    d = torch.empty(len(a) + shift, dtype=torch.int32, device="cuda")
    d[shift:] = torch.from_numpy(np.ascontiguousarray(a)).cuda()
    return d[shift:]


def _dimension(rng, n, kind):
    keys = (rng.permutation(2 * n)[:n] + 5).astype(np.int32)
    return dict(key=keys, val=rng.integers(1, 50, n).astype(np.int32) if kind % 2 else None,
                flt=rng.integers(0, 6, n).astype(np.int32) if kind < 2 else None,
                mode=[L.MB_FILTER_EQ, L.MB_FILTER_EQ_OR_EQ][kind % 2], slots=2 * n + 3, kmin=4)


@pytest.mark.parametrize("n", [1, 7, 8, 9, 2_047, 2_048, 2_049, 100_001])
@pytest.mark.parametrize("shift", [0, 1])
def test_tables_together(n, shift):
    rng = np.random.default_rng(n + shift)
    dims = [_dimension(rng, max(1, n // (k + 1)), k) for k in range(4)]
    arr, out, keep = (L.MbTableBuild * 4)(), [], []
    for b, d in zip(arr, dims):
        words = d["slots"] * (2 if d["val"] is not None else 1)
        ht = torch.full((words + 4,), 77, dtype=torch.int32, device="cuda")[2 * shift:][:words]
        bits = torch.full(((d["slots"] + 31) // 32,), -1, dtype=torch.int32, device="cuda")
        cols = [None if d[k] is None else _dev(d[k], shift) for k in ("flt", "key", "val")]
        b.filter_col, b.dim_key, b.dim_val = (ssb._p(c) for c in cols)
        b.filter_mode, b.c1, b.c2 = d["mode"], 1, 3
        b.num_tuples, b.ht, b.num_slots, b.key_min, b.presence = len(d["key"]), ht.data_ptr(), d["slots"], d["kmin"], \
            bits.data_ptr()
        out.append((ht, bits))
        keep.append(cols)
    zero = torch.full((1_003 + shift,), 9, dtype=torch.int32, device="cuda")
    L.device_status(0)
    L.call("mb_build_tables", arr, 4, zero[shift:].data_ptr(), 1_001, ssb._stream())
    torch.cuda.synchronize()
    z = zero.cpu().numpy()
    assert (z[:shift] == 9).all() and (z[shift: shift + 1_001] == 0).all() and (z[shift + 1_001:] == 9).all()
    for (ht, bits), d in zip(out, dims):
        layout = L.MB_HT_KEY if d["val"] is None else L.MB_HT_KEY_VAL
        ref = np.zeros(ht.numel(), np.int32)
        O.build_ht(d["flt"], d["mode"], 1, 3, d["key"], d["val"], ref, d["slots"], d["kmin"], layout)
        assert np.array_equal(ht.cpu().numpy(), ref)
        on = ref != 0 if layout == L.MB_HT_KEY else ref.reshape(-1, 2).any(1)
        packed = np.zeros(bits.numel() * 32, np.uint8)
        packed[: d["slots"]] = on
        assert np.array_equal(bits.cpu().numpy(), np.packbits(packed, bitorder="little").view(np.int32))
    assert L.device_status(0) == 0


@pytest.mark.parametrize("n", [5, 300_003])
def test_builds_into_one_table_keep_their_order(n):
    """Three builds into one table (or its bitmap alone), a fourth into another between them: rows
    of a later build replace the payloads of an earlier one's, and the first key stays."""
    rng = np.random.default_rng(n)
    slots = 2 * n + 3
    dims = [_dimension(rng, n, 1) for _ in range(4)]
    tables = [torch.full((2 * slots,), 7, dtype=torch.int32, device="cuda") for _ in range(2)]
    bits = torch.full(((slots + 31) // 32,), -1, dtype=torch.int32, device="cuda")
    cols = [[_dev(d[k]) for k in ("flt", "key", "val")] for d in dims]
    arr = (L.MbTableBuild * 4)()
    into = [0, 1, 0, 0]
    for b, c, d, k in zip(arr, cols, dims, into):
        b.filter_col, b.dim_key, b.dim_val = (ssb._p(x) for x in c)
        b.filter_mode, b.c1, b.c2 = d["mode"], 1, 3
        b.num_tuples, b.ht, b.num_slots, b.key_min = n, tables[k].data_ptr(), slots, d["kmin"]
        b.presence = bits.data_ptr() if k == 0 else None
    L.call("mb_build_tables", arr, 4, None, 0, ssb._stream())
    torch.cuda.synchronize()
    ref = [np.zeros(2 * slots, np.int32) for _ in range(2)]
    for d, k in zip(dims, into):
        O.build_ht(d["flt"], d["mode"], 1, 3, d["key"], d["val"], ref[k], slots, d["kmin"], L.MB_HT_KEY_VAL)
    for t, r in zip(tables, ref):
        assert np.array_equal(t.cpu().numpy(), r)
    packed = np.zeros(bits.numel() * 32, np.uint8)
    packed[:slots] = ref[0].reshape(-1, 2).any(1)
    assert np.array_equal(bits.cpu().numpy(), np.packbits(packed, bitorder="little").view(np.int32))


@pytest.mark.parametrize("n", [1, 9, 2_049, 300_003])
@pytest.mark.parametrize("shift", [0, 1])
def test_single_build_of_columns(n, shift):
    rng = np.random.default_rng(n)
    d = _dimension(rng, n, 1)
    ht = torch.zeros(2 * d["slots"], dtype=torch.int32, device="cuda")
    cols = [_dev(d[k], shift) for k in ("flt", "key", "val")]
    L.call("mb_build_pht", cols[0].data_ptr(), d["mode"], 1, 3, cols[1].data_ptr(), cols[2].data_ptr(), n, ht.data_ptr(),
           d["slots"], d["kmin"], None, ssb._stream())
    ref = np.zeros(2 * d["slots"], np.int32)
    O.build_ht(d["flt"], d["mode"], 1, 3, d["key"], d["val"], ref, d["slots"], d["kmin"], L.MB_HT_KEY_VAL)
    assert np.array_equal(ht.cpu().numpy(), ref)


def test_refused_arguments():
    ht = torch.zeros(8, dtype=torch.int32, device="cuda")
    arr = (L.MbTableBuild * 1)()
    arr[0].ht, arr[0].num_slots, arr[0].num_tuples = ht.data_ptr(), 8, 3  # rows without a key column
    with pytest.raises(L.MbError):
        L.call("mb_build_tables", arr, 1, None, 0, ssb._stream())
    with pytest.raises(L.MbError):
        L.call("mb_build_tables", arr, 9, None, 0, ssb._stream())
