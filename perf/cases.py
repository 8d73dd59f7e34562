"""The work this library's users have it do, as cases that can be timed and checked.

A case names a kind of work and its sizes:

* ``filter_aggregate`` — the q11 form: three range filters, one sum (``ssb.q11``).
* ``query_a`` / ``query_b`` — whole star queries, hash-table builds and fused probe
  (``ssb.query_a``, ``ssb.query_b``).
* ``engine`` — a query of the executor through the segment cache: the engine's builds, then
  ``mb_probe_group_by_GPU2`` (or ``mb_filter_probe_group_by_GPU2``) over a segment list.
* ``split`` — split execution on one device: ``mb_filter_probe_GPU2`` selects rows into an
  offset list, the host reads its length, ``mb_probe_group_by_GPU3`` finishes the query.
* ``list`` — ``mb_probe_group_by_GPU3`` over an offset list that arrived from elsewhere (the
  CPU half of a split query).
* ``batch`` — many queries in one scan: a prepared ``BatchPlan``, or ``run_batch`` with its
  planning, as a server that meets new queries on each launch calls it.
* ``planner_forward`` / ``planner_train`` — the learned planner: predictions for a window of
  (query, segment) pairs, and one training step (gradients, then Adam).

Columns are drawn here with seeded generators on the GPU, with the star schema's ranges and
value distributions; ``exact`` computes each answer from them with plain 64-bit torch.
"""
import ctypes as C
import math

import numpy as np
import torch

from mordred_b200 import _lib as L
from mordred_b200 import batch as B
from mordred_b200 import ssb

SEG = 1 << 20
YEARS = 7
NATIONS = 25
BRANDS = 1000

# Dimension rows of the star schema at scale factors 1 and 20 (supplier, customer, part).
DIMS_SF1 = (2_000, 30_000, 200_000)
DIMS_SF20 = (40_000, 600_000, 1_000_000)


def _star(kind, rows, dims=DIMS_SF20, **more):
    return dict(kind=kind, rows=rows, s_len=dims[0], c_len=dims[1], p_len=dims[2], **more)


def listed():
    return [
        # the smallest filter-aggregate in use: one scale-factor-1 fact table
        dict(_star("filter_aggregate", 6_000_000), name="filter_aggregate_6M"),
        # the same scan over a table far beyond L2: bandwidth alone
        dict(_star("filter_aggregate", 120_000_000), name="filter_aggregate_120M"),
        # the two headline star queries at scale factor 20, builds included
        dict(_star("query_a", 120_000_000), name="query_a_120M"),
        dict(_star("query_b", 120_000_000), name="query_b_120M"),
        # an interactive query over one segment and a ragged tail: builds and launches count
        dict(_star("query_b", 1_050_001), name="query_b_1M"),
        # the executor's form of Query B: 23 shuffled cache segments, the last one ragged
        dict(_star("engine", 22 * SEG + 931_201, filters=0, wide_groups=False), name="engine_23seg"),
        # the GPU selects and its list goes on to a second operator: both halves of a split query
        dict(_star("split", 22 * SEG + 931_201, filters=1), name="split_23seg"),
        # a list the CPU half selected: two million rows scattered over 23 segments
        dict(_star("list", 22 * SEG + 931_201, entries=2_000_003), name="list_2M"),
        # a full batch of mixed queries over a resident table
        dict(_star("batch", 60_000_000, queries=256, date_sorted=False, planned=True), name="batch_256"),
        # one launch of the serving loop: one chunk of the date-sorted table and the queries on it
        dict(_star("batch", 75_000_000, queries=24, date_sorted=True, planned=False), name="batch_24_serving"),
        # placement of a whole window of queries: one prediction per (query, segment) pair
        dict(kind="planner_forward", samples=1_700_000, name="planner_forward_1700k"),
        # one training step of the planner at its batch size
        dict(kind="planner_train", samples=256, name="planner_train_256"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["filter_aggregate", "query_a", "query_b", "engine", "split", "list", "batch",
                       "planner_forward", "planner_train"])
    if kind == "planner_forward":
        return dict(kind=kind, samples=_log_uniform(rng, 64, 1_700_000))
    if kind == "planner_train":
        return dict(kind=kind, samples=_log_uniform(rng, 64, 4_096))
    dims = tuple(_log_uniform(rng, lo, hi) for lo, hi in zip(DIMS_SF1, DIMS_SF20))
    if kind in ("filter_aggregate", "query_a", "query_b"):
        lo = 1_000_000 if kind == "filter_aggregate" else 300_000
        return _star(kind, _log_uniform(rng, lo, 120_000_000), dims)
    rows = _log_uniform(rng, 700_000, 23 * SEG)
    if kind == "engine":
        return _star(kind, rows, dims, filters=rng.choice([0, 2]), wide_groups=rng.random() < 0.3)
    if kind == "split":
        return _star(kind, rows, dims, filters=rng.choice([0, 1, 2]))
    if kind == "list":
        return _star(kind, rows, dims, entries=max(1_000, int(rows * rng.uniform(0.001, 0.2))))
    rows = _log_uniform(rng, 1_000_000, 60_000_000)
    return _star(kind, rows, dims, queries=_log_uniform(rng, 2, 256), date_sorted=rng.random() < 0.5,
                 planned=rng.random() < 0.5)


# ---- inputs --------------------------------------------------------------------------------

def _generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7919 + 17)
    return g


def _uniform(g, lo, hi, n):
    """n int32 values, uniform in [lo, hi]."""
    return torch.randint(lo, hi + 1, (n,), dtype=torch.int32, device="cuda", generator=g)


def _calendar():
    return torch.tensor(B.CALENDAR, dtype=torch.int32, device="cuda")


def _dimensions(case, g):
    cal = _calendar()
    t = {"d_datekey": cal, "d_year": cal // 10_000}
    for x, n in (("s", case["s_len"]), ("c", case["c_len"])):
        city = _uniform(g, 0, 249, n)
        t.update({f"{x}_city": city, f"{x}_nation": city // 10, f"{x}_region": city // 50})
    t["s_suppkey"] = torch.arange(1, case["s_len"] + 1, dtype=torch.int32, device="cuda")
    t["c_custkey"] = torch.arange(1, case["c_len"] + 1, dtype=torch.int32, device="cuda")
    t["p_partkey"] = torch.arange(1, case["p_len"] + 1, dtype=torch.int32, device="cuda")
    t["p_brand1"] = _uniform(g, 0, BRANDS - 1, case["p_len"])
    t["p_category"] = t["p_brand1"] // 40
    t["p_mfgr"] = t["p_brand1"] // 200
    return t


RANGES = {"lo_quantity": (1, 50), "lo_discount": (0, 10), "lo_extendedprice": (90_100, 10_494_950),
          "lo_revenue": (90_100, 10_494_950), "lo_supplycost": (54_000, 600_000)}


def _fact(case, g, names):
    """Fact columns by name, drawn in the order asked for."""
    n, out = case["rows"], {}
    keys = {"lo_suppkey": (1, case["s_len"]), "lo_custkey": (1, case["c_len"]), "lo_partkey": (1, case["p_len"])}
    for name in names:
        if name == "lo_orderdate":
            if case.get("date_sorted"):
                day = (torch.arange(n, device="cuda") * len(B.CALENDAR)) // n
            else:
                day = _uniform(g, 0, len(B.CALENDAR) - 1, n)
            out[name] = _calendar()[day]
        else:
            lo, hi = keys.get(name) or RANGES[name]
            out[name] = _uniform(g, lo, hi, n)
    return out


def _sizes(case):
    return ssb.Sizes(lo_len=case["rows"], s_len=case["s_len"], c_len=case["c_len"], p_len=case["p_len"])


FACT = {"filter_aggregate": ssb.Q11_COLUMNS, "query_a": ssb.QA_FACT, "query_b": ssb.QB_FACT,
        "engine": ssb.QB_FACT + ["lo_quantity", "lo_discount"], "split": ssb.QB_FACT + ["lo_quantity"],
        "list": ssb.QB_FACT, "batch": B.BATCH_FACT}

# The engine's filters: quantity in [5, 40] (and discount in [1, 6]); split: orderdate, quantity.
ENGINE_FILTERS = [("lo_quantity", 5, 40), ("lo_discount", 1, 6)]
SPLIT_FILTERS = [("lo_orderdate", 19930601, 19970630), ("lo_quantity", 5, 40)]


def _tables(case, seed):
    """Dimension and fact columns of a star case; both prepare() and exact() start here."""
    g = _generator(seed)
    t = _dimensions(case, g)
    t.update(_fact(case, g, FACT[case["kind"]]))
    return t


def _listed_rows(case, seed):
    """`entries` different fact rows in ascending order, spread over the table."""
    n, k = case["rows"], min(case["entries"], case["rows"])
    g = _generator(seed + 1_000_003)
    step = n // k
    base = torch.arange(k, device="cuda", dtype=torch.int64) * n // k
    return (base + torch.randint(0, step, (k,), device="cuda", generator=g)).to(torch.int32)


def _batch_ranges(case, seed):
    """Mixed queries, the three templates in turn: selectivity log-uniform in [1e-5, 0.3], part
    of it carried by the small-domain predicates and the rest by a range of orderdates."""
    rng = np.random.default_rng(seed)
    domains = {"agg": [("discount", 0, 10), ("quantity", 1, 50)], "qa": [("s_region", 0, 4), ("category", 0, 24)],
               "qb": [("c_region", 0, 4), ("s_region", 0, 4), ("mfgr", 0, 4)]}
    cal, out = B.CALENDAR, []

    def pick(lo, hi, width):
        width = max(1, min(hi - lo + 1, width))
        start = lo + int(rng.integers(0, hi - lo + 2 - width))
        return start, start + width - 1

    for k in range(case["queries"]):
        template = ("agg", "qa", "qb")[k % 3]
        sel = math.exp(rng.uniform(math.log(1e-5), math.log(0.3)))
        parts = rng.uniform(0.0, 0.8) * rng.dirichlet(np.ones(len(domains[template])))
        got, q = 1.0, {"template": template}
        for (name, lo, hi), part in zip(domains[template], parts):
            width = max(1, int(round((hi - lo + 1) * sel ** part)))
            got *= width / (hi - lo + 1)
            q[name] = pick(lo, hi, width)
        a, b = pick(0, len(cal) - 1, int(round(len(cal) * sel / got)))
        q["date"] = (cal[a], cal[b])
        out.append(q)
    return out


# ---- the engine's segment cache and tables -------------------------------------------------------

def _cache(t, names, rows, seed):
    """The columns cut into segments scattered over a pool of cache slots, each column's slot
    per segment, and a shuffled segment list that ends with the ragged segment."""
    rng = np.random.default_rng(seed)
    nseg = (rows + SEG - 1) // SEG
    slots = rng.permutation(nseg * len(names)).reshape(len(names), nseg)
    pool = torch.zeros(nseg * len(names) * SEG, dtype=torch.int32, device="cuda")
    idx = {}
    for i, name in enumerate(names):
        for s in range(nseg):
            part = t[name][s * SEG: min(rows, (s + 1) * SEG)]
            at = int(slots[i, s]) * SEG
            pool[at: at + part.numel()] = part
        idx[name] = torch.from_numpy(slots[i].astype(np.int32)).cuda()
    order = np.concatenate([rng.permutation(nseg - 1), [nseg - 1]]).astype(np.int16)
    return pool, idx, torch.from_numpy(order).cuda()


# name -> key, payload column of narrow / wide groups, filter column, filter mode and constants
def _engine_dims(case):
    wide = case.get("wide_groups", False)
    return [("s", "s_suppkey", "s_nation" if wide else None, "s_region", L.MB_FILTER_EQ, 1, 0, case["s_len"], 0),
            ("c", "c_custkey", None if wide else "c_nation", "c_region", L.MB_FILTER_EQ, 1, 0, case["c_len"], 0),
            ("p", "p_partkey", "p_category" if wide else None, "p_mfgr", L.MB_FILTER_EQ_OR_EQ, 0, 1, case["p_len"], 0),
            ("d", "d_datekey", "d_year", None, 0, 0, 0, ssb.DATE_SLOTS, ssb.DATE_MIN)]


def _group_multipliers(case):
    """Group multipliers of supplier, customer, part, date and the group count."""
    if case.get("wide_groups", False):  # year x supplier nation x category
        return (YEARS * 25, 0, YEARS, 1), YEARS * NATIONS * 25
    return (0, YEARS, 0, 1), YEARS * NATIONS  # year x customer nation


def _engine_build(st):
    for k, ht in st["ht"].items():
        ht.zero_()
        f, b, n = st["builds"][k]
        L.call("mb_build_GPU2", None, C.byref(f), C.byref(b), n, ht.data_ptr(), 0, None, ssb._stream())


def _engine_state(case, seed, names):
    t = _tables(case, seed)
    pool, idx, order = _cache(t, names, case["rows"], seed)
    dims = {k: v for k, v in t.items() if not k.startswith("lo_")}
    del t
    mul, groups = _group_multipliers(case)
    ht, builds = {}, {}
    p = lambda name: dims[name].data_ptr() if name else None
    for k, key, val, flt, mode, c1, c2, slots, kmin in _engine_dims(case):
        ht[k] = torch.zeros(2 * slots, dtype=torch.int32, device="cuda")
        builds[k] = (L.MbFilterArgsGPU(p(flt), None, c1, c2, 0, 0, mode, 0),
                     L.MbBuildArgsGPU(p(key), p(val), slots, kmin, 0), dims[key].numel())
    return dict(case=case, pool=pool, idx=idx, order=order, dims=dims, ht=ht, builds=builds, mul=mul, groups=groups,
                res=torch.zeros(6 * groups, dtype=torch.int32, device="cuda"))


KEYS = {"s": "lo_suppkey", "c": "lo_custkey", "p": "lo_partkey", "d": "lo_orderdate"}


def _probe_args(st, case, which):
    """Engine probes of the dimensions in `which`; the others are absent."""
    slots = {"s": case["s_len"], "c": case["c_len"], "p": case["p_len"], "d": ssb.DATE_SLOTS}
    return L.MbProbeArgsGPU(*(st["idx"][KEYS[k]].data_ptr() if k in which else None for k in "scpd"),
                            *(st["ht"][k].data_ptr() if k in which else None for k in "scpd"),
                            *(slots[k] if k in which else 0 for k in "scpd"), 0, 0, 0, ssb.DATE_MIN)


def _filter_args(st, filters):
    col = lambda i: st["idx"][filters[i][0]].data_ptr() if len(filters) > i else None
    const = [c for _, lo, hi in filters for c in (lo, hi)] + [0] * (4 - 2 * len(filters))
    return L.MbFilterArgsGPU(col(0), col(1), *const, L.MB_FILTER_BETWEEN, L.MB_FILTER_BETWEEN)


def _groupby_args(st, group_cols):
    """SUM(revenue - supplycost); group_cols: the dimension columns read at listed dimension rows."""
    return L.MbGroupbyArgsGPU(st["idx"]["lo_revenue"].data_ptr(), st["idx"]["lo_supplycost"].data_ptr(), *group_cols,
                              0, 0, 0, 1992, *st["mul"], st["groups"], 0)


# ---- prepare / run -----------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    return PREPARE[kind](case, seed)


def run(state):
    return RUN[state["case"]["kind"]](state)


def _prepare_star(case, seed):
    return dict(case=case, t=_tables(case, seed), ws=ssb.StarWorkspace(_sizes(case)))


def _run_filter_aggregate(st):
    rev = ssb.q11(st["t"], st["case"]["rows"], st["ws"])
    return rev, st["ws"]["cnt"]


def _run_query_a(st):
    return ssb.query_a(st["t"], st["ws"])


def _run_query_b(st):
    return ssb.query_b(st["t"], st["ws"])


def _prepare_engine(case, seed):
    filters = ENGINE_FILTERS[: case["filters"]]
    names = ssb.QB_FACT + [f[0] for f in filters]
    st = _engine_state(case, seed, names)
    st["probe"] = _probe_args(st, case, "scpd")
    st["group"] = _groupby_args(st, (None, None, None, None))
    st["filter"] = _filter_args(st, filters)
    return st


def _run_engine(st):
    case = st["case"]
    _engine_build(st)
    st["res"].zero_()
    tail = (case["rows"], st["res"].data_ptr(), 0, st["order"].data_ptr(), ssb._stream())
    if case["filters"]:
        L.call("mb_filter_probe_group_by_GPU2", st["pool"].data_ptr(), C.byref(st["filter"]), C.byref(st["probe"]),
               C.byref(st["group"]), *tail)
    else:
        L.call("mb_probe_group_by_GPU2", st["pool"].data_ptr(), C.byref(st["probe"]), C.byref(st["group"]), *tail)
    return st["res"]


def _prepare_split(case, seed):
    filters = SPLIT_FILTERS[: case["filters"]]
    names = ssb.QB_FACT + [f[0] for f in filters if f[0] not in ssb.QB_FACT]
    st = _engine_state(case, seed, names)
    _engine_build(st)  # the dimension side of the query ran before
    n = case["rows"]
    st["off"] = [torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(3)]
    st["total"] = torch.zeros(1, dtype=torch.int32, device="cuda")
    lo, s, c = (x.data_ptr() for x in st["off"])
    st["list"] = L.MbOffsetGPU(lo, s, c, None, None)
    st["filter"] = _filter_args(st, filters)
    st["select_probe"] = _probe_args(st, case, "sc")
    st["probe"] = _probe_args(st, case, "pd")
    # the customer's nation at the listed customer row; its column is one cache segment long
    st["nation"], st["pool"] = _append_dimension(st["pool"], st["dims"]["c_nation"])
    st["group"] = _groupby_args(st, (None, st["nation"].data_ptr(), None, None))
    return st


def _append_dimension(pool, col):
    """A dimension column as one more segment of the cache pool; (its slot array, the pool)."""
    slot = pool.numel() // SEG
    out = torch.zeros(pool.numel() + SEG, dtype=torch.int32, device="cuda")
    out[: pool.numel()] = pool
    out[pool.numel(): pool.numel() + col.numel()] = col
    return torch.tensor([slot], dtype=torch.int32, device="cuda"), out


def _run_split(st):
    case = st["case"]
    st["total"].zero_()
    st["res"].zero_()
    pool, stream = st["pool"].data_ptr(), ssb._stream()
    if case["filters"]:
        L.call("mb_filter_probe_GPU2", pool, C.byref(st["filter"]), C.byref(st["select_probe"]), C.byref(st["list"]),
               case["rows"], st["total"].data_ptr(), 0, st["order"].data_ptr(), stream)
    else:
        L.call("mb_probe_GPU2", pool, C.byref(st["select_probe"]), C.byref(st["list"]), case["rows"],
               st["total"].data_ptr(), 0, st["order"].data_ptr(), stream)
    found = int(st["total"].item())  # the host needs the list's length to go on with it
    L.call("mb_probe_group_by_GPU3", pool, C.byref(st["list"]), C.byref(st["probe"]), C.byref(st["group"]), found,
           st["res"].data_ptr(), stream)
    return st["res"], found


def _prepare_list(case, seed):
    t = _tables(case, seed)
    rows = _listed_rows(case, seed)
    cust = t["lo_custkey"][rows.long()] - 1  # the customer row each listed row joined with
    del t
    st = _engine_state(case, seed, ssb.QB_FACT)
    _engine_build(st)
    st["off"] = [rows, cust]
    st["list"] = L.MbOffsetGPU(rows.data_ptr(), None, cust.data_ptr(), None, None)
    st["probe"] = _probe_args(st, case, "pd")
    st["nation"], st["pool"] = _append_dimension(st["pool"], st["dims"]["c_nation"])
    st["group"] = _groupby_args(st, (None, st["nation"].data_ptr(), None, None))
    return st


def _run_list(st):
    st["res"].zero_()
    L.call("mb_probe_group_by_GPU3", st["pool"].data_ptr(), C.byref(st["list"]), C.byref(st["probe"]),
           C.byref(st["group"]), st["off"][0].numel(), st["res"].data_ptr(), ssb._stream())
    return st["res"]


def _prepare_batch(case, seed):
    t = _tables(case, seed)
    st = dict(case=case, t=t, pats=B.build_pats(t, _sizes(case)))
    st["queries"] = [B.Query(**q) for q in _batch_ranges(case, seed)]
    st["flat"], st["results"] = B.result_buffers(st["queries"])
    if case["planned"]:
        st["plan"] = B.BatchPlan(t, st["pats"], st["queries"], st["results"], case["rows"])
    return st


def _run_batch(st):
    st["flat"].zero_()
    if "plan" in st:
        st["plan"].run()
    else:
        B.run_batch(st["t"], st["pats"], st["queries"], st["results"], st["case"]["rows"])
    return st["flat"].view(torch.int64)


def _planner_inputs(case, seed, targets):
    """He-initialised parameters with small biases, standardised features, targets near the
    log milliseconds of real segments; for training, Adam's moments some way into a run."""
    g = _generator(seed)
    normal = lambda *shape: torch.randn(shape, device="cuda", generator=g)
    i, h, o = L.MB_MLP_IN, L.MB_MLP_HIDDEN, L.MB_MLP_OUT
    parts = []
    for a, b in ((i, h), (h, h), (h, o)):
        parts += [normal(a * b) * math.sqrt(2.0 / a), normal(b) * 0.1]
    st = dict(case=case, params=torch.cat(parts), x=normal(case["samples"], i))
    if targets:
        st["target"] = normal(case["samples"], o) * 1.5 - 0.5
        st["m"] = normal(L.MB_MLP_PARAMS) * 1e-2
        st["v"] = normal(L.MB_MLP_PARAMS).square() * 1e-3 + 1e-4
        st["g"] = torch.zeros(L.MB_MLP_PARAMS, device="cuda")
        st["loss"] = torch.zeros(1, device="cuda")
        st["step"] = 1000
    else:
        st["y"] = torch.empty(case["samples"], o, device="cuda")
    return st


def _run_planner_forward(st):
    L.call("mb_mlp_forward", st["params"].data_ptr(), st["x"].data_ptr(), st["case"]["samples"], st["y"].data_ptr(),
           ssb._stream())
    return st["y"]


ADAM = dict(lr=1e-3, beta1=0.9, beta2=0.999, eps=1e-8, weight_decay=1e-5)


def _run_planner_train(st):
    stream = ssb._stream()
    st["g"].zero_()
    st["loss"].zero_()
    st["step"] += 1
    L.call("mb_mlp_backward", st["params"].data_ptr(), st["x"].data_ptr(), st["target"].data_ptr(),
           st["case"]["samples"], st["g"].data_ptr(), st["loss"].data_ptr(), stream)
    L.call("mb_mlp_adam", st["params"].data_ptr(), st["g"].data_ptr(), st["m"].data_ptr(), st["v"].data_ptr(),
           L.MB_MLP_PARAMS, ADAM["lr"], ADAM["beta1"], ADAM["beta2"], ADAM["eps"], st["step"], ADAM["weight_decay"],
           stream)
    return {"params": st["params"], "grads": st["g"], "m": st["m"], "v": st["v"], "loss": st["loss"]}


PREPARE = {"filter_aggregate": _prepare_star, "query_a": _prepare_star, "query_b": _prepare_star,
           "engine": _prepare_engine, "split": _prepare_split, "list": _prepare_list, "batch": _prepare_batch,
           "planner_forward": lambda case, seed: _planner_inputs(case, seed, False),
           "planner_train": lambda case, seed: _planner_inputs(case, seed, True)}
RUN = {"filter_aggregate": _run_filter_aggregate, "query_a": _run_query_a, "query_b": _run_query_b,
       "engine": _run_engine, "split": _run_split, "list": _run_list, "batch": _run_batch,
       "planner_forward": _run_planner_forward, "planner_train": _run_planner_train}


# ---- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    kind, n = case["kind"], case.get("rows", case.get("samples"))
    if kind.startswith("planner"):
        macs = L.MB_MLP_IN * L.MB_MLP_HIDDEN + L.MB_MLP_HIDDEN ** 2 + L.MB_MLP_HIDDEN * L.MB_MLP_OUT
        p = 4 * L.MB_MLP_PARAMS
        if kind == "planner_forward":
            return {"bytes": p + n * 4 * (L.MB_MLP_IN + L.MB_MLP_OUT), "flops": 2 * macs * n}
        # forward, input gradients of the two upper layers, weight gradients; p, m, v in and out, grads out
        return {"bytes": 7 * p + n * 4 * (L.MB_MLP_IN + L.MB_MLP_OUT),
                "flops": 2 * n * (3 * macs - L.MB_MLP_IN * L.MB_MLP_HIDDEN)}
    s, c, p, d = case["s_len"], case["c_len"], case["p_len"], ssb.DATE_SLOTS
    if kind == "filter_aggregate":
        return {"bytes": 16 * n + 12, "flops": 0}
    if kind == "query_a":  # dimension columns in, tables out
        return {"bytes": 16 * n + 8 * s + 12 * p + 4 * s + 8 * p + 8 * d + 16 * ssb.QA_GROUPS, "flops": 0}
    if kind == "query_b":
        return {"bytes": 24 * n + 8 * s + 12 * c + 8 * p + 4 * s + 8 * c + 4 * p + 8 * d + 16 * ssb.QB_GROUPS,
                "flops": 0}
    tables = 8 * (s + c + p + d)
    if kind == "engine":
        return {"bytes": (24 + 4 * case["filters"]) * n + tables + 12 * (s + c + p) + 24 * _group_multipliers(case)[1],
                "flops": 0}
    if kind == "split":
        # filter columns and the two probed keys of every row; the list written and read; part
        # and date keys and the two aggregate columns of the selected rows
        kept = n / 25
        kept *= (1, 1492 / 2557, 1492 / 2557 * 36 / 50)[case["filters"]]
        return {"bytes": int((8 + 4 * case["filters"]) * n + kept * (12 + 8 + 16)) + tables, "flops": 0}
    if kind == "list":
        return {"bytes": min(case["entries"], n) * (8 + 16) + 8 * (p + d) + 4 * c, "flops": 0}
    return {"bytes": 36 * n + 4 * (s + c + p + d) + 16 * ssb.QA_GROUPS * case["queries"] // 3, "flops": 0}


# ---- the same answers from plain 64-bit torch ------------------------------------------------------

CHUNK = 1 << 24


def _chunks(n):
    return [(a, min(n, a + CHUNK)) for a in range(0, n, CHUNK)]


def _pack(stride, groups, keys, counts, sums):
    """int32 [stride * groups]: key columns of the groups that have rows, then the 64-bit sum."""
    out = torch.zeros(groups, stride, dtype=torch.int32, device="cuda")
    seen = counts > 0
    for slot, col in keys.items():
        out[:, slot] = torch.where(seen, col, torch.zeros_like(col)).to(torch.int32)
    out[:, stride - 2:] = sums.view(torch.int32).view(groups, 2)
    return out.view(-1)


def _accumulate(sums, counts, group, value):
    sums.index_add_(0, group, value)
    counts.index_add_(0, group, torch.ones_like(value))


def _member(t, rows, key, lut):
    return lut[t[key][rows].long() - 1]


def _year(t, rows):
    return (t["lo_orderdate"][rows] // 10_000).long() - 1992


def _exact_filter_aggregate(case, seed):
    t = _tables(case, seed)
    rev = torch.zeros((), dtype=torch.int64, device="cuda")
    cnt = torch.zeros((), dtype=torch.int64, device="cuda")
    for a, b in _chunks(case["rows"]):
        disc, qty = t["lo_discount"][a:b], t["lo_quantity"][a:b]
        od = t["lo_orderdate"][a:b]
        first = (disc >= 1) & (disc <= 3) & (qty < 25)
        cnt += first.sum()
        ok = first & (od > 19930000) & (od < 19940000)
        rev += (t["lo_extendedprice"][a:b].long() * disc.long())[ok].sum()
    return rev.view(1), cnt.to(torch.int32).view(1)


def _group_grid(*sizes):
    """The value of each mixed-radix digit over the group index, first digit fastest."""
    g = torch.arange(math.prod(sizes), device="cuda")
    out = []
    for n in sizes:
        out.append(g % n)
        g = g // n
    return out


def _exact_query_a(case, seed):
    t = _tables(case, seed)
    s_ok, p_ok, brand = t["s_region"] == 1, t["p_category"] == 1, t["p_brand1"].long()
    groups = YEARS * BRANDS
    sums, counts = (torch.zeros(groups, dtype=torch.int64, device="cuda") for _ in range(2))
    for a, b in _chunks(case["rows"]):
        rows = slice(a, b)
        ok = _member(t, rows, "lo_suppkey", s_ok) & _member(t, rows, "lo_partkey", p_ok)
        rows = a + ok.nonzero().view(-1)
        _accumulate(sums, counts, _member(t, rows, "lo_partkey", brand) * YEARS + _year(t, rows),
                    t["lo_revenue"][rows].long())
    y, br = _group_grid(YEARS, BRANDS)
    return _pack(4, groups, {0: y + 1992, 1: br}, counts, sums)


def _query_b_rows(t, rows, parts=True):
    """Which of `rows` join: supplier and customer region 1, and (parts) mfgr 0 or 1."""
    ok = _member(t, rows, "lo_suppkey", t["s_region"] == 1) & _member(t, rows, "lo_custkey", t["c_region"] == 1)
    if parts:
        ok &= _member(t, rows, "lo_partkey", t["p_mfgr"] <= 1)
    return ok


def _exact_nation_groups(case, seed, stride, keep):
    """SUM(revenue - supplycost) by (year, customer nation) over the rows keep(t, a, b) gives."""
    t = _tables(case, seed)
    groups = YEARS * NATIONS
    sums, counts = (torch.zeros(groups, dtype=torch.int64, device="cuda") for _ in range(2))
    for a, b in _chunks(case["rows"]):
        rows = keep(t, a, b)
        _accumulate(sums, counts, _member(t, rows, "lo_custkey", t["c_nation"].long()) * YEARS + _year(t, rows),
                    t["lo_revenue"][rows].long() - t["lo_supplycost"][rows].long())
    y, nat = _group_grid(YEARS, NATIONS)
    keys = {0: y + 1992, 1: nat} if stride == 4 else {1: nat, 3: y + 1992}
    return _pack(stride, groups, keys, counts, sums)


def _exact_query_b(case, seed):
    return _exact_nation_groups(case, seed, 4, lambda t, a, b: a + _query_b_rows(t, slice(a, b)).nonzero().view(-1))


def _passes(t, rows, filters):
    ok = torch.ones_like(t["lo_orderdate"][rows], dtype=torch.bool)
    for name, lo, hi in filters:
        ok &= (t[name][rows] >= lo) & (t[name][rows] <= hi)
    return ok


def _exact_engine(case, seed):
    filters = ENGINE_FILTERS[: case["filters"]]
    keep = lambda t, a, b: a + (_query_b_rows(t, slice(a, b)) & _passes(t, slice(a, b), filters)).nonzero().view(-1)
    if not case["wide_groups"]:
        return _exact_nation_groups(case, seed, 6, keep)
    t = _tables(case, seed)
    groups = YEARS * 25 * NATIONS
    sums, counts = (torch.zeros(groups, dtype=torch.int64, device="cuda") for _ in range(2))
    for a, b in _chunks(case["rows"]):
        rows = keep(t, a, b)
        group = (_member(t, rows, "lo_suppkey", t["s_nation"].long()) * 25 +
                 _member(t, rows, "lo_partkey", t["p_category"].long())) * YEARS + _year(t, rows)
        _accumulate(sums, counts, group, t["lo_revenue"][rows].long() - t["lo_supplycost"][rows].long())
    y, cat, nat = _group_grid(YEARS, 25, NATIONS)
    return _pack(6, groups, {0: nat, 2: cat, 3: y + 1992}, counts, sums)


def _exact_split(case, seed):
    found = 0

    def keep(t, a, b):
        nonlocal found
        ok = _query_b_rows(t, slice(a, b), parts=False) & _passes(t, slice(a, b), SPLIT_FILTERS[: case["filters"]])
        found += int(ok.sum())
        ok &= _member(t, slice(a, b), "lo_partkey", t["p_mfgr"] <= 1)
        return a + ok.nonzero().view(-1)

    res = _exact_nation_groups(case, seed, 6, keep)
    return res, found


def _exact_list(case, seed):
    listed_rows = _listed_rows(case, seed).long()

    def keep(t, a, b):
        rows = listed_rows[(listed_rows >= a) & (listed_rows < b)]
        return rows[_member(t, rows, "lo_partkey", t["p_mfgr"] <= 1)]

    return _exact_nation_groups(case, seed, 6, keep)


def _exact_batch(case, seed):
    t = _tables(case, seed)
    out = []
    for q in _batch_ranges(case, seed):
        within = lambda v, r: (v >= r[0]) & (v <= r[1])
        agg, qa = q["template"] == "agg", q["template"] == "qa"
        groups = 1 if agg else YEARS * (BRANDS if qa else NATIONS)
        sums, counts = (torch.zeros(groups, dtype=torch.int64, device="cuda") for _ in range(2))
        for a, b in _chunks(case["rows"]):
            rows = a + within(t["lo_orderdate"][a:b], q["date"]).nonzero().view(-1)
            if agg:
                rows = rows[within(t["lo_discount"][rows], q["discount"]) & within(t["lo_quantity"][rows], q["quantity"])]
                sums += (t["lo_extendedprice"][rows].long() * t["lo_discount"][rows].long()).sum()
                continue
            rows = rows[_member(t, rows, "lo_suppkey", within(t["s_region"], q["s_region"]))]
            if qa:
                rows = rows[_member(t, rows, "lo_partkey", within(t["p_category"], q["category"]))]
                major, value = _member(t, rows, "lo_partkey", t["p_brand1"].long()), t["lo_revenue"][rows].long()
            else:
                rows = rows[_member(t, rows, "lo_custkey", within(t["c_region"], q["c_region"]))]
                rows = rows[_member(t, rows, "lo_partkey", within(t["p_mfgr"], q["mfgr"]))]
                major = _member(t, rows, "lo_custkey", t["c_nation"].long())
                value = t["lo_revenue"][rows].long() - t["lo_supplycost"][rows].long()
            _accumulate(sums, counts, major * YEARS + _year(t, rows), value)
        if agg:
            out.append(sums)
        else:
            y, major = _group_grid(YEARS, groups // YEARS)
            out.append(_pack(4, groups, {0: y + 1992, 1: major}, counts, sums).view(torch.int64))
    return torch.cat(out)


def _layers(params):
    i, h, o = L.MB_MLP_IN, L.MB_MLP_HIDDEN, L.MB_MLP_OUT
    out, at = [], 0
    for shape in ((i, h), (h,), (h, h), (h,), (h, o), (o,)):
        n = math.prod(shape)
        out.append(params[at: at + n].view(shape))
        at += n
    return out


def _mlp(params, x):
    w1, b1, w2, b2, w3, b3 = _layers(params)
    return torch.relu(torch.relu(x @ w1 + b1) @ w2 + b2) @ w3 + b3


def _exact_planner_forward(case, seed):
    st = _planner_inputs(case, seed, False)
    return _mlp(st["params"].double(), st["x"].double())


def _exact_planner_train(case, seed):
    st = _planner_inputs(case, seed, True)
    params = st["params"].double().requires_grad_(True)
    diff = _mlp(params, st["x"].double()) - st["target"].double()
    loss = 0.5 * diff.square().sum()
    (grads,) = torch.autograd.grad(loss / case["samples"], params)
    p, m, v, step = params.detach(), st["m"].double(), st["v"].double(), st["step"] + 1
    g = grads + ADAM["weight_decay"] * p
    m = ADAM["beta1"] * m + (1 - ADAM["beta1"]) * g
    v = ADAM["beta2"] * v + (1 - ADAM["beta2"]) * g * g
    mhat, vhat = m / (1 - ADAM["beta1"] ** step), v / (1 - ADAM["beta2"] ** step)
    p = p - ADAM["lr"] * mhat / (vhat.sqrt() + ADAM["eps"])
    return {"params": p, "grads": grads, "m": m, "v": v, "loss": loss.detach().view(1)}


EXACT = {"filter_aggregate": _exact_filter_aggregate, "query_a": _exact_query_a, "query_b": _exact_query_b,
         "engine": _exact_engine, "split": _exact_split, "list": _exact_list, "batch": _exact_batch,
         "planner_forward": _exact_planner_forward, "planner_train": _exact_planner_train}


def exact(case, seed):
    return EXACT[case["kind"]](case, seed)
