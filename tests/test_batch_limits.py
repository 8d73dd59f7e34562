"""Batches at the limits of the planner — end points and shared memory run out — sized by
mb_batch_workspace_bytes and checked against a plain numpy evaluation of every query."""
import numpy as np
import pytest

import test_batch_masks as M
from mordred_b200 import _lib as L
from mordred_b200 import batch as B

pytestmark = pytest.mark.gpu


def _check(n, queries, seed, ranges=(), **launch):
    """`ranges`: fact columns drawn anew, (name, values)."""
    t, words = M._data(n, seed, 0.9)
    rng = np.random.default_rng(seed + 1)
    for name, values in ranges:
        t[name] = rng.integers(0, values, n).astype(np.int64)
    L.device_status(0)
    got = M._run(t, words, queries, n, **launch)
    for i, (q, g) in enumerate(zip(queries, got)):
        assert M._same(q, g, M._expected(q, t, words)), (i, q)
    assert L.device_status(0) == 0


@pytest.mark.parametrize("count", [200, 256])
def test_more_end_points_than_fit_named_in_different_orders(count):
    """Two wide attributes with more than 768 end points together. The first query is of a class
    of its own and names the quantity; the others, the largest class, name the part first."""
    part, quantity = B.F(L.MB_COL_DIM_P, 5, 10), B.FACT["lo_quantity"]
    grouped = dict(layout=L.MB_RES_CRYSTAL4, keys=[(B.F(L.MB_COL_DIM_D, 0, 4), 0, 1)], op=L.MB_AGG_SUM,
                   agg=[B.FACT["lo_revenue"]], total=16, dims=12)
    queries = [dict(layout=L.MB_RES_SCALAR, keys=[], op=L.MB_AGG_SUB, agg=[B.FACT["lo_revenue"], B.FACT["lo_supplycost"]],
                    total=1, dims=0, preds=[(quantity, 0, 3_999)])]
    for i in range(1, count):
        queries.append(dict(grouped, preds=[(part, i, 1_023 - i), (quantity, 2 * i, 3_999 - 3 * i)]))
    _check(7_001, queries, count, ranges=[("lo_quantity", 4_000)])


@pytest.mark.parametrize("smem", [-1, 0, 131_072])
@pytest.mark.parametrize("count", [16, 40])
def test_more_group_counts_than_shared_memory_holds(count, smem):
    """Every query has a group count of its own, near 1,000: most get no shared-memory sums."""
    year, brand = B.F(L.MB_COL_DIM_D, 0, 4), B.F(L.MB_COL_DIM_P, 4, 6)
    queries = [dict(layout=[L.MB_RES_DENSE, L.MB_RES_CRYSTAL4][i % 2], keys=[(year, 0, 1), (brand, 0, 16)],
                    op=L.MB_AGG_SUB, agg=[B.FACT["lo_revenue"], B.FACT["lo_supplycost"]], total=1_024 - i, dims=15,
                    preds=[(B.FACT["lo_quantity"], i % 7, 49), (B.FACT["lo_discount"], -3, 13 - i % 5)])
               for i in range(count)]
    _check(5_003, queries, count, smem_group_bytes=smem)


@pytest.mark.parametrize("count,values,launch", [
    (256, 416, {}), (200, 488, {}), (256, 512, {}), (64, 512, dict(threads=512, items_per_thread=4)),
    (128, 512, dict(threads=512, items_per_thread=4)), (256, 512, dict(threads=512, items_per_thread=4, stages=8))])
def test_more_tables_than_shared_memory_holds(count, values, launch):
    """Eight attributes of many values and all nine fact columns: a smaller launch, and tables
    left in the workspace."""
    fields = [B.F(M.DIM_COL[k], shift, 9) for k in "SCPD" for shift in (0, 9)]
    aggs = [(L.MB_AGG_SUB, ["lo_revenue", "lo_supplycost"]), (L.MB_AGG_MUL, ["lo_extendedprice", "lo_discount"]),
            (L.MB_AGG_SUM, ["lo_quantity"])]
    rng = np.random.default_rng(count)
    queries = []
    for i in range(count):
        layout = [L.MB_RES_SCALAR, L.MB_RES_CRYSTAL4, L.MB_RES_DENSE][i % 3]
        keys = [] if layout == L.MB_RES_SCALAR else [(B.F(L.MB_COL_DIM_D, 0, 4), 0, 1), (B.F(L.MB_COL_DIM_S, 4, 3), 0, 16)]
        preds = [(fields[i % 8], 0, values - 1)]
        for f in rng.permutation(8)[: int(rng.integers(0, 4))]:
            lo = int(rng.integers(0, values))
            preds.append((fields[f], lo, int(rng.integers(lo, values))))
        op, agg = aggs[i % 3]
        queries.append(dict(layout=layout, keys=keys, op=op, agg=[B.FACT[a] for a in agg], total=130, dims=i % 16,
                            preds=preds))
    _check(6_401, queries, count + values, **launch)


@pytest.mark.parametrize("n", [1_535, 1_536, 1_537, 768 * 148, 768 * 148 + 1, 1_536 * 148 + 5])
@pytest.mark.parametrize("count", [24, 64])
def test_default_launches_of_few_rows(n, count):
    """Up to a tile of 768 rows an SM, and more."""
    M._check(n, M._queries(count, n, 3), n)
