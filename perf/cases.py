"""Timed workloads of the query path, from the smallest single query to the 600M-row shared batch.

Each case is one call that a program makes on tables it has resident on the GPU:

* ``query``  -- ``Database.execute``: one query, its result words read back to the host;
* ``stream`` -- ``ExecCtx.execute`` (cx_execute): one query enqueued on the caller's stream, its
  result left in the caller's device buffers, as a C++ executor or the request loop drives it;
* ``batch``  -- ``Database.execute_shared``: a batch of template queries over one shared scan;
* ``finish`` -- cx_finalize: a grouped aggregate buffer into ordered result rows on the device;
* ``compact`` -- cx_compact_sparse: the non-zero group tuples of a sparse result.

Tables are the seeded synthetic star schema of ``practice_b200.datagen``, generated on the device.
"""
from __future__ import annotations

import random

import torch

from practice_b200 import _lib, datagen, queries
from practice_b200.engine import SHARED_DEFAULT, Database, make_tuning

NULLS = {"lo_revenue": 100, "c_city": 50}  # permille of NULL values, as the nullable Q3.1 configuration has them

# Fact columns each query shape reads; `commit` shapes also read lo_commitdate.
FACT_COLS = {"q11": queries.Q11_COLS, "q31": queries.Q31_COLS, "q31n": queries.Q31_COLS}
EXPANDING = {"or_year": queries.or_join_year, "or_filter": queries.or_join_then_filter,
             "mht_tier": queries.mht_year_tier, "mht_supp": queries.mht_then_supplier, "mht_brand": queries.mht_brand}
# Launch shapes: the library's default, and the two that the autotuner picks most for join and scan-only shapes.
TUNINGS = {"default": {}, "compact": dict(compact=1), "compact64": dict(compact=2),
           "ring": dict(block_threads=512, items_per_thread=8, stages=4, bitmap_budget=0)}


def listed():
    return [
        # Latency of the smallest interactive query: launches and the result's way back, hardly any rows.
        dict(name="q11_60k", kind="query", shape="q11", rows=60_011, tuning="default"),
        # The configured Q1.1 workload: 6M rows, a scalar SUM behind a date join.
        dict(name="q11_6m", kind="query", shape="q11", rows=6_000_000, tuning="default"),
        # The configured Q3.1 workload: three joins, 4,375 groups, 60M rows.
        dict(name="q31_60m", kind="stream", shape="q31", rows=60_000_000, tuning="compact"),
        # Its nullable variant: three-valued filters, validity bitmaps, three aggregates.
        dict(name="q31n_60m", kind="stream", shape="q31n", rows=60_000_000, tuning="compact"),
        # One dashboard template over the whole benchmark table as its own kernel.
        dict(name="t3_600m", kind="stream", shape="t3", rows=600_000_000, tuning="compact"),
        # The headline: a 32-query batch over 600M rows, results read back.
        dict(name="batch32_600m", kind="batch", rows=600_000_000, queries=32, path="cube"),
        # A short queue on a small ragged table: the shared path's launch cost.
        dict(name="batch6_6m", kind="batch", rows=5_999_987, queries=6, path="cube"),
        # The per-query mask path, taken by batches whose attributes have no usable ranges.
        dict(name="masks16_60m", kind="batch", rows=60_000_000, queries=16, path="masks"),
        # OR-join over two date keys, then a filter and MIN / MAX / AVG over a nullable column.
        dict(name="or_filter_60m", kind="stream", shape="or_filter", rows=60_000_000, tuning="default"),
        # Multi-value hash join into 35,000 (brand, year, tier) groups; an odd table size.
        dict(name="mht_brand_30m", kind="stream", shape="mht_brand", rows=30_000_001, tuning="default"),
        # ORDER BY over up to 62,500 (city, city) groups on the device.
        dict(name="finish_city", kind="finish", shape="city", rows=2_000_000, limit=0),
        # Compaction of a many-group sparse result (8.25M group slots, 330 MB).
        dict(name="compact_wide", kind="compact", rows=6_000_000, noalloc=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["query", "stream", "stream", "stream", "batch", "batch", "finish", "compact"])
    if kind == "query":
        shape = rng.choice(["q11", "q31", "t0", "t1", "t2"])
        return dict(kind=kind, shape=shape, rows=_log_int(rng, 50_000, 12_000_000), tuning="default", literals=rng.randrange(1000))
    if kind == "stream":
        shape = rng.choice(["q31", "q31n", "t1", "t2", "t3", "or_year", "or_filter", "mht_tier", "mht_supp", "mht_brand"])
        if shape in EXPANDING:
            return dict(kind=kind, shape=shape, rows=_log_int(rng, 1_000_000, 60_000_000), tuning="default")
        return dict(kind=kind, shape=shape, rows=_log_int(rng, 1_000_000, 300_000_000),
                    tuning=rng.choice(["default", "compact", "compact64"]), literals=rng.randrange(1000))
    if kind == "batch":
        path = rng.choice(["cube", "cube", "masks"])
        return dict(kind=kind, rows=_log_int(rng, 1_000_000, 200_000_000 if path == "cube" else 60_000_000),
                    queries=rng.randint(5, 32), path=path)
    if kind == "finish":
        return dict(kind=kind, shape=rng.choice(["q31", "city"]), rows=_log_int(rng, 20_000, 6_000_000),
                    limit=rng.choice([0, 10, 1000]))
    return dict(kind=kind, rows=_log_int(rng, 100_000, 12_000_000), noalloc=rng.random() < 0.5)


def _plan(case):
    """The case's query; a program keeps its text, so literals do not depend on the data's seed."""
    shape, n = case["shape"], case["rows"]
    if shape in EXPANDING:
        return EXPANDING[shape](n)
    rng = random.Random(case.get("literals", 7))
    if shape[0] == "t":
        return queries.template(int(shape[1]), rng, n)
    if shape == "city":
        plan = queries.city_pairs(rng, n)
        plan.order_by = [(0, False), (2, True)]
        return plan
    if shape == "q11":
        return queries.ssb_q11(n)
    return queries.ssb_q31_nullable(n) if shape == "q31n" else queries.ssb_q31(n)


def _plans(case, seed):
    """A batch's queries: a mix of the templates, every one among them, with fresh constants per request."""
    mix, rng = random.Random(case["queries"]), random.Random(seed)
    return [queries.template(i if i < 4 else mix.randrange(4), rng, case["rows"]) for i in range(case["queries"])]


def _database(case, seed, plans):
    fact = sorted({c for p in plans for c in p.columns_read()})
    dims = tuple(t for t in ("DDATE", "CUSTOMER", "SUPPLIER", "PART", "PARTSUPP")
                 if any(s.dim == t for p in plans for kind, s in p.steps if kind == "join"))
    nullable = {c for p in plans for c in p.nullable}
    db = Database(0)
    generated = sorted((set(fact) - {"lo_commitdate"}) | ({"lo_orderdate"} if "lo_commitdate" in fact else set()))
    db.generate_ssb(case["rows"], seed, generated, nulls={c: k for c, k in NULLS.items() if c in nullable}, dims=dims)
    if "lo_commitdate" in fact:
        # The order date plus 0..90 days.
        gen = torch.Generator(device=db.device).manual_seed(seed)
        days = torch.from_numpy(datagen.DATE_KEYS).to(db.device)
        ext = torch.from_numpy(datagen.EXT_DATE_KEYS).to(db.device)
        commit = torch.empty(case["rows"], dtype=torch.int32, device=db.device)
        for r in range(0, case["rows"], 1 << 24):
            at = torch.searchsorted(days, db.cols["lo_orderdate"][r:r + (1 << 24)])
            at += torch.randint(0, datagen.COMMIT_LAG_DAYS, at.shape, generator=gen, device=db.device)
            commit[r:r + at.numel()] = ext[at]
        db.load_column("LINEORDER", "lo_commitdate", commit)
    return db


def _stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        plans = _plans(case, seed)
        db = _database(case, seed, plans)
        tuning = make_tuning(**{**SHARED_DEFAULT, **({"cube": 0} if case["path"] == "masks" else {})})
        db.shared_program(plans, tuning)
        return dict(kind=kind, db=db, plans=plans, tuning=tuning)
    if kind == "compact":
        plan = queries.wide_groups(random.Random(7), case["rows"])
    else:
        plan = _plan(case)
    db = _database(case, seed, [plan])
    tuning = make_tuning(**TUNINGS[case["tuning"]]) if TUNINGS.get(case.get("tuning")) else None
    module = db.compile(plan, tuning)
    if kind == "query":
        return dict(kind=kind, db=db, plan=plan, tuning=tuning)
    res, val = db.alloc_result(module)
    for table, n in db.rows.items():
        db.ctx.set_rows(table, n)
    db.ctx.set_result(res.data_ptr(), res.numel(), val.data_ptr(), val.numel())
    state = dict(kind=kind, db=db, plan=plan, module=module, res=res, val=val)
    if kind == "stream":
        return state
    # finish / compact: the aggregate buffer that the query leaves.
    db.ctx.execute(module, _stream())
    db.ctx.sync()
    groups = plan.group_slots
    if kind == "finish":
        from practice_b200 import results

        cap = max(groups, 1)
        state.update(cap=cap, limit=case["limit"] or None, types=results.column_types(plan),
                     nullable=results.output_nullable(plan),
                     cols=torch.zeros(plan.visible_ts * cap, dtype=torch.int64, device=db.device),
                     cval=torch.zeros(plan.visible_ts * ((cap + 63) // 64), dtype=torch.int64, device=db.device))
    else:
        state.update(dst=torch.zeros_like(res), count=torch.zeros(1, dtype=torch.int64, device=db.device),
                     fn=_lib.lib.cx_compact_sparse_noalloc if case["noalloc"] else _lib.lib.cx_compact_sparse)
    # The tables are not read again.
    db.reset()
    return state


def run(state):
    kind, db = state["kind"], state["db"]
    if kind == "query":
        got = db.execute(state["plan"], state["tuning"])
        return got.words.view("int64"), got.validity.view("int64"), got.kernel_error
    if kind == "stream":
        db.ctx.execute(state["module"], _stream())
        return state["res"], state["val"]
    if kind == "batch":
        got = db.execute_shared(state["plans"], state["tuning"])
        return [r.words.view("int64") for r in got], [r.validity.view("int64") for r in got]
    plan = state["plan"]
    if kind == "finish":
        n = _lib.finalize(state["res"].data_ptr(), state["val"].data_ptr(), plan.group_slots, plan.storage_ts,
                          state["types"], state["nullable"], plan.sparse, not plan.groups, list(plan.order_by),
                          state["limit"], state["cols"].data_ptr(), state["cval"].data_ptr(), state["cap"], _stream())
        # The rows asked for (past the last row both buffers stay as they were).
        return n, state["cols"].view(plan.visible_ts, -1)[:, :state["limit"]], state["cval"]
    _lib.check(state["fn"](state["res"].data_ptr(), plan.group_slots, plan.storage_ts, state["dst"].data_ptr(),
                           state["count"].data_ptr(), _stream()), "compaction")
    return state["dst"], state["count"]


def _column_rows(plan):
    """Every column a plan reads -> rows of its table."""
    fact = {c: plan.fact.rows for c in plan.columns_read()}
    for kind, s in plan.steps:
        if kind != "join":
            continue
        cols = [s.pk] + (s.filter.columns() if s.filter is not None else []) + ([s.payload] if s.payload else [])
        for c in cols + list(s.gathers):
            fact.setdefault(c, datagen.DIM_ROWS[s.dim])
    return fact


def work(case):
    kind = case["kind"]
    if kind == "batch":
        plans = _plans(case, 0)
    elif kind == "compact":
        plans = [queries.wide_groups(random.Random(7), case["rows"])]
    else:
        plans = [_plan(case)]
    words = sum(p.group_slots * p.storage_ts for p in plans)
    if kind in ("finish", "compact"):
        # The buffer and its validity bits read once; the rows that come out are at most as many as the fact rows.
        out = min(words, case["rows"] * plans[0].storage_ts)
        return {"bytes": words * 8 + (words / 8 if kind == "finish" else 0) + out * 8, "flops": 0}
    cols = {}
    for p in plans:
        cols.update(_column_rows(p))
    nullable = {c for p in plans for c in p.nullable}
    read = sum(n * 4 + (n / 8 if c in nullable else 0) for c, n in cols.items())
    return {"bytes": read + words * 8 + words / 8, "flops": 0}


def exact(case, seed):
    """Every output is whole numbers (64-bit sums, counts, keys and bits), compared as they are."""
    return None
