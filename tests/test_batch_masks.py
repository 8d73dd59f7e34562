"""The batched kernel's masks, classes and match lists at their edges, against a plain numpy
evaluation of every query: batch sizes around the mask words, more classes than the kernel
keeps, more matches than a list holds, dimension rows that are missing or read without being
required, values outside every query's hull, all result layouts, and tile remainders."""
import ctypes as C

import numpy as np
import pytest
import torch

from mordred_b200 import _lib as L
from mordred_b200 import batch as B
from mordred_b200 import ssb

pytestmark = pytest.mark.gpu
SLOTS = {"S": 40, "C": 70, "P": 90, "D": 61}
KEYCOL = {"S": "lo_suppkey", "C": "lo_custkey", "P": "lo_partkey", "D": "lo_orderdate"}
DIM_COL = {"S": L.MB_COL_DIM_S, "C": L.MB_COL_DIM_C, "P": L.MB_COL_DIM_P, "D": L.MB_COL_DIM_D}


def _data(n, seed, present):
    rng = np.random.default_rng(seed)
    t = {"lo_orderdate": rng.integers(0, 61, n), "lo_quantity": rng.integers(0, 50, n),
         "lo_discount": rng.integers(-3, 14, n), "lo_extendedprice": rng.integers(-2**31, 2**31, n),
         "lo_suppkey": rng.integers(0, 80, n), "lo_custkey": rng.integers(0, 140, n),
         "lo_partkey": rng.integers(0, 400, n), "lo_revenue": rng.integers(0, 10**7, n),
         "lo_supplycost": rng.integers(0, 10**6, n)}
    t = {k: v.astype(np.int64) for k, v in t.items()}
    words = {}
    for k, slots in SLOTS.items():
        w = rng.integers(0, 2**18, slots).astype(np.int64) | (1 << 31)
        w[rng.random(slots) > present] = 0
        words[k] = w
    return t, words


def _field(code, t, words):
    col, shift, width = code >> 11, (code >> 6) & 31, code & 63
    if col < L.MB_NUM_FACT_COLS:
        v = t[B.BATCH_FACT[col]]
    else:
        k = "SCPD"[col - L.MB_COL_DIM_S]
        v = words[k][t[KEYCOL[k]] % SLOTS[k]]
    return v if width == 32 else (v >> shift) & ((1 << width) - 1)


def _wrap(v):
    return (v + 2**31) % 2**32 - 2**31


def _expected(q, t, words):
    n = len(t["lo_quantity"])
    ok = np.ones(n, bool)
    for code, lo, hi in q["preds"]:
        v = _field(code, t, words)
        ok &= (v >= lo) & (v <= hi)
    for i, k in enumerate("SCPD"):
        if q["dims"] >> i & 1:
            ok &= words[k][t[KEYCOL[k]] % SLOTS[k]] != 0
    a = [_field(c, t, words)[ok] for c in q["agg"]]
    val = _wrap(a[0] if q["op"] == L.MB_AGG_SUM else a[0] - a[1] if q["op"] == L.MB_AGG_SUB else a[0] * a[1])
    keys = [_field(c, t, words)[ok] for c, _, _ in q["keys"]]
    if q["layout"] == L.MB_RES_SCALAR:
        return np.array([val.sum()], np.int64)
    g = _wrap(sum((k - mn) * mul for k, (_, mn, mul) in zip(keys, q["keys"])) + np.zeros(len(val), np.int64))
    g = np.fmod(g, q["total"])  # the remainder has the sign of the index; a negative one drops the row
    q["bad"] = bool((g < 0).any())
    keys, val, g = [k[g >= 0] for k in keys], val[g >= 0], g[g >= 0]
    sums = np.zeros(q["total"], np.int64)
    np.add.at(sums, g, val)
    if q["layout"] == L.MB_RES_DENSE:
        return sums
    # keys of different rows can wrap onto one group, which then shows one row's: all pairs
    pairs = {}
    for i, h in enumerate(g):
        pairs.setdefault(int(h), set()).add(tuple(int(k[i]) for k in keys))
    return sums, pairs


def _same(q, got, exp):
    if q["layout"] != L.MB_RES_CRYSTAL4:
        return np.array_equal(got, exp)
    sums, pairs = exp
    got = got.reshape(-1, 4)
    if not np.array_equal(np.ascontiguousarray(got[:, 2:]).view(np.int64).reshape(-1), sums):
        return False
    return all(tuple(got[h, : len(q["keys"])]) in pairs.get(h, {(0,) * len(q["keys"])}) and
               not got[h, len(q["keys"]): 2].any() for h in range(q["total"]))


def _run(t, words, queries, n, **launch):
    dt = {k: torch.from_numpy(v.astype(np.int32)).cuda() for k, v in t.items()}
    dw = {k: torch.from_numpy(v.astype(np.uint32).view(np.int32)).cuda() for k, v in words.items()}
    res, arr = [], (L.MbBatchQuery * len(queries))()
    for c, q in zip(arr, queries):
        scalar = q["layout"] == L.MB_RES_SCALAR
        crystal = q["layout"] == L.MB_RES_CRYSTAL4
        res.append(torch.zeros(1 if scalar else q["total"] * (2 if crystal else 1), dtype=torch.int64, device="cuda"))
        c.num_preds = len(q["preds"])
        for i, p in enumerate(q["preds"]):
            c.pred_field[i], c.pred_lo[i], c.pred_hi[i] = p
        c.dims_required, c.agg_op = q["dims"], q["op"]
        for i, f in enumerate(q["agg"]):
            c.agg_field[i] = f
        c.num_keys, c.total_val, c.res_layout, c.res = len(q["keys"]), q["total"], q["layout"], res[-1].data_ptr()
        for i, (f, mn, mul) in enumerate(q["keys"]):
            c.key_field[i], c.key_min[i], c.key_mul[i] = f, mn, mul
    a = L.MbBatchArgs()
    a.num_rows = n
    for i, name in enumerate(B.BATCH_FACT):
        a.fact[i] = dt[name].data_ptr()
    for i, k in enumerate("SCPD"):
        a.dim[i] = L.MbPat(dw[k].data_ptr(), SLOTS[k], 0)
    a.num_queries, a.queries = len(queries), C.cast(arr, C.POINTER(L.MbBatchQuery))
    a.smem_group_bytes = -1
    for k, v in launch.items():
        setattr(a, k, v)
    ws = torch.empty(max(16, int(L.lib().mb_batch_workspace_bytes(C.byref(a)))), dtype=torch.uint8, device="cuda")
    a.workspace, a.workspace_bytes = ws.data_ptr(), ws.numel()
    L.check("mb_batch_run", L.lib().mb_batch_run(C.byref(a), ssb._stream()))
    torch.cuda.synchronize()
    out = []
    for q, r in zip(queries, res):
        r = r.cpu().numpy()
        out.append(r.view(np.int32) if q["layout"] == L.MB_RES_CRYSTAL4 else r)
    return out


FACT_FIELDS = [(B.FACT["lo_orderdate"], 0, 60), (B.FACT["lo_quantity"], 0, 49), (B.FACT["lo_discount"], -3, 13)]
DIM_FIELDS = [(B.F(DIM_COL[k], s, w), 0, 2**w - 1) for k, s, w in
              (("S", 0, 3), ("C", 3, 4), ("P", 5, 5), ("D", 2, 2))]


def _queries(count, seed, classes, wide=False, dims_only=False):
    """Random queries of `classes` aggregate forms over three fact and four dimension attributes."""
    rng = np.random.default_rng(seed)
    forms = []
    for i in range(classes):
        layout = [L.MB_RES_SCALAR, L.MB_RES_CRYSTAL4, L.MB_RES_DENSE][i % 3]
        keys = [] if layout == L.MB_RES_SCALAR else \
            [(B.F(DIM_COL["D"], 0, 4), 3, 1), (B.F(DIM_COL["P"], 4, 3), 0, 16 + i)][: 1 + i % 2]
        forms.append(dict(layout=layout, keys=keys, op=[L.MB_AGG_MUL, L.MB_AGG_SUB, L.MB_AGG_SUM][i % 3],
                          agg=[B.FACT["lo_revenue"], B.FACT["lo_supplycost"]][: 1 if i % 3 == 2 else 2],
                          total=1 if layout == L.MB_RES_SCALAR else [137, 1500][(i // 3) % 2] + i,
                          dims=int(rng.integers(0, 16))))
    out = []
    for k in range(count):
        q = dict(forms[k % classes])
        fields = (DIM_FIELDS if dims_only else FACT_FIELDS + DIM_FIELDS)
        q["preds"] = []
        for f in rng.permutation(len(fields))[: int(rng.integers(0, 4))]:
            code, lo, hi = fields[f]
            a = int(rng.integers(lo, hi + 1))
            b = hi if wide else int(rng.integers(a - 1, hi + 1))  # also empty ranges
            q["preds"].append((code, lo if wide else a, b))
        out.append(q)
    return out


def _check(n, queries, seed, present=0.8, **launch):
    t, words = _data(n, seed, present)
    L.device_status(0)
    got = _run(t, words, queries, n, **launch)
    for i, (q, g) in enumerate(zip(queries, got)):
        assert _same(q, g, _expected(q, t, words)), (i, q)
    assert L.device_status(0) == (L.MB_STATUS_GROUP_RANGE if any(q.get("bad") for q in queries) else 0)


@pytest.mark.parametrize("count", [1, 32, 33, 64, 65, 128, 129, 256])
def test_mask_words(count):
    _check(9_001, _queries(count, count, 3), count)


@pytest.mark.parametrize("classes", [1, 4, 5, 11])
@pytest.mark.parametrize("count", [40, 200])
def test_classes(classes, count):
    _check(5_000, _queries(count, classes, classes), classes)


@pytest.mark.parametrize("count,classes", [(48, 2), (250, 1), (250, 6)])
def test_more_matches_than_a_list_holds(count, classes):
    _check(4_100, _queries(count, 5, classes, wide=True), 5, present=1.0)


@pytest.mark.parametrize("count", [20, 100])
@pytest.mark.parametrize("present", [0.0, 0.3])
def test_missing_dimension_rows(count, present):
    _check(6_007, _queries(count, 9, 3, dims_only=True), 9, present=present)


@pytest.mark.parametrize("n", [1, 767, 768, 959, 960, 961, 1535, 1536, 1537])
@pytest.mark.parametrize("count", [24, 70])
def test_tile_remainders(n, count):
    _check(n, _queries(count, n, 3), n)


@pytest.mark.parametrize("threads,items", [(256, 4), (512, 4), (512, 2), (768, 1), (768, 2), (960, 1)])
@pytest.mark.parametrize("count", [30, 60, 100, 240])
def test_rows_per_lane(threads, items, count):
    _check(8_200, _queries(count, count, 4), count, threads=threads, items_per_thread=items)
