"""Per-query mask scan (cube = 0) against the oracle, each query alone, where its
parts change: 1, 32, 33 and 64 queries (one and two mask words), all of one shape
(bits past a word), ragged and tiny tables, tables that lie in shared memory with
32 copies of a word, with one, or not at all, COUNT and SUM mixed, values of both
signs, a group key or value that holds a literal, values outside the filter
windows, and consecutive row ranges with unaligned column starts."""
import random

import numpy as np
import pytest

import oracle
from practice_b200 import datagen, queries
from practice_b200.engine import SHARED_DEFAULT, make_tuning
from practice_b200.plan import Group, PlanBuilder, col, lit, star

pytestmark = pytest.mark.gpu

COLS = sorted(set(queries.BATCH_COLS) | {"lo_extendedprice"})
DIMS = ("DDATE", "CUSTOMER", "SUPPLIER", "PART")


@pytest.fixture(scope="module")
def db():
    from practice_b200.engine import Database
    return Database(0)


def load(db, n):
    ht = datagen.host_tables(31 + n % 7, n, COLS)
    rng = np.random.default_rng(n)
    ht.columns["lo_revenue"] = rng.integers(-2**31, 2**31, n).astype(np.int32)
    ht.columns["lo_discount"] = rng.integers(-300, 300, n).astype(np.int32)  # more values than a filter window
    db.reset()
    db.load_host_tables(ht, datagen.ssb_tables(n, COLS))
    return ht


def shapes(n, rng):
    t = datagen.ssb_tables(n, COLS)

    def b(name):
        return PlanBuilder(t, "LINEORDER", name=name)

    def scalar():
        p = b("s")
        p.filter(col("lo_discount").ge(rng.randint(-310, 0)))
        p.filter(col("lo_quantity").lt(rng.randint(1, 60)))
        return p.aggregate([], [("sum", col("lo_revenue") * col("lo_discount")), ("count", star()), ("sum", col("lo_supplycost"))])

    def few():
        p = b("f")
        p.join("DDATE", "lo_orderdate", where=col("d_year").ge(rng.randint(1992, 1999)))
        p.filter(col("lo_discount").lt(rng.randint(-300, 310)))
        return p.aggregate([queries._g("d_year")], [("sum", col("lo_revenue"))])

    def some():
        p = b("m")
        p.join("SUPPLIER", "lo_suppkey", where=col("s_region").le(rng.randint(0, 4)))
        p.join("CUSTOMER", "lo_custkey", where=col("c_region").ge(rng.randint(0, 4)))
        p.filter((col("lo_quantity") + col("lo_discount")).lt(rng.randint(-200, 200)))  # a residual filter
        return p.aggregate([queries._g("c_nation"), queries._g("s_region")], [("count", star()), ("sum", col("lo_revenue") - col("lo_supplycost"))])

    def many():
        p = b("l")
        p.join("PART", "lo_partkey", where=col("p_mfgr").le(rng.randint(0, 4)))
        p.join("DDATE", "lo_orderdate", where=col("d_month").le(rng.randint(1, 12)))
        return p.aggregate([queries._g("p_brand1"), queries._g("d_month")], [("sum", col("lo_supplycost"))])

    def literal():
        p = b("v")
        p.filter(col("lo_quantity").ge(rng.randint(1, 50)))
        return p.aggregate([Group(col("lo_quantity"), 1, 50, False)], [("sum", col("lo_revenue") * lit(rng.randint(-5, 5)))])

    return [scalar, few, some, many, literal]


def check(db, ht, plans, results):
    rows = {"LINEORDER": ht.fact_rows, **{d: datagen.DIM_ROWS[d] for d in DIMS}}
    for p, got in zip(plans, results):
        ref = oracle.run_plan(p.text(), ht.columns, ht.validity, rows, p.group_slots * p.storage_ts)
        assert got.kernel_error == 0 and got.timing.mode == 0
        np.testing.assert_array_equal(got.words, ref.words, err_msg=p.name)
        np.testing.assert_array_equal(got.validity, ref.validity, err_msg=p.name)


@pytest.mark.parametrize("n", [1, 63, 65, 60_011])
@pytest.mark.parametrize("nq", [1, 32, 33, 64])
@pytest.mark.parametrize("kw", [dict(), dict(block_threads=256)], ids=str)
def test_mixed_batches(db, n, nq, kw):
    ht = load(db, n)
    rng = random.Random(nq)
    makers = shapes(n, rng)
    plans = [makers[i % len(makers)]() for i in range(nq)]
    check(db, ht, plans, db.execute_shared(plans, make_tuning(**{**SHARED_DEFAULT, "cube": 0, **kw})))


@pytest.mark.parametrize("k", range(5))
def test_one_shape_past_a_word(db, k):
    ht = load(db, 30_001)
    plans = [shapes(30_001, random.Random(100 + i))[k]() for i in range(40)]
    check(db, ht, plans, db.execute_shared(plans, make_tuning(**{**SHARED_DEFAULT, "cube": 0})))


def test_row_ranges(db):
    """Ranges that start at odd rows: columns no longer aligned for vector loads."""
    n = 50_003
    ht = load(db, n)
    rng = random.Random(9)
    plans = [m() for m in shapes(n, rng) for _ in range(2)]
    prog = db.shared_program(plans, make_tuning(**{**SHARED_DEFAULT, "cube": 0}))
    qs, params, bufs = db.shared_prepare(prog, plans)
    for t, r in db.rows.items():
        db.ctx.set_rows(t, r)
    stream = db.torch.cuda.current_stream().cuda_stream
    at = 0
    for size in (1, 17_001, 20_000, n):
        db.ctx.shared_execute_rows(prog.module, qs, params, at, size, [at > 0] * len(qs), stream)
        db.ctx.sync()
        at = min(n, at + size)
    rows = {"LINEORDER": n, **{d: datagen.DIM_ROWS[d] for d in DIMS}}
    for p, (res, val, words) in zip(plans, bufs):
        ref = oracle.run_plan(p.text(), ht.columns, ht.validity, rows, p.group_slots * p.storage_ts)
        np.testing.assert_array_equal(res.cpu().numpy().view(np.uint64)[:words], ref.words, err_msg=p.name)
        np.testing.assert_array_equal(val.cpu().numpy().view(np.uint64)[:(words + 63) // 64], ref.validity, err_msg=p.name)
