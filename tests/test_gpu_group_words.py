"""Shared-memory group tables of 32-bit words (SUM as low and high word, COUNT,
MIN / MAX of an int32 column) against the oracle, bit for bit: values of both
signs and at the ends of int32, so that carries cross the words and negative
minima and maxima keep the unsigned 64-bit order; NULLs; 11 to 3,850 groups, so
that a word has 32 copies, a few or one; block sizes that change the copies;
rows merged by group first; and a multi-value join, whose counts take two words."""
import numpy as np
import pytest

import oracle
from practice_b200 import datagen, queries
from practice_b200.engine import make_tuning
from practice_b200.plan import Group, PlanBuilder, col, star

pytestmark = pytest.mark.gpu

COLS = sorted(set(queries.BATCH_COLS) | set(queries.OR_COLS) | set(queries.MHT_COLS))
DIMS = ("DDATE", "CUSTOMER", "SUPPLIER", "PART", "PARTSUPP")
N = 120_011


@pytest.fixture(scope="module")
def loaded():
    from practice_b200.engine import Database
    db = Database(0)
    ht = datagen.host_tables(77, N, COLS, {"lo_revenue": 150}, dims=DIMS)
    rng = np.random.default_rng(5)
    ends = np.array([-2**31, -2**31 + 1, -1, 0, 1, 2**31 - 1], dtype=np.int32)
    signed = rng.integers(-2**31, 2**31, N).astype(np.int32)
    ht.columns["lo_revenue"] = np.where(rng.random(N) < 0.2, rng.choice(ends, N), signed).astype(np.int32)
    ht.columns["lo_supplycost"] = np.where(rng.random(N) < 0.5, np.int32(-1), signed[::-1]).astype(np.int32)
    db.load_host_tables(ht, datagen.ssb_tables(N, COLS))
    return db, ht


def check(loaded, plan, tuning):
    db, ht = loaded
    rows = {"LINEORDER": N, **{d: datagen.DIM_ROWS[d] for d in DIMS}}
    ref = oracle.run_plan(plan.text(), ht.columns, ht.validity, rows, plan.group_slots * plan.storage_ts)
    got = db.execute(plan, tuning)
    assert got.kernel_error == 0
    fw = len(got.words)
    np.testing.assert_array_equal(got.words, ref.words[:fw])
    np.testing.assert_array_equal(got.validity, ref.validity[: (fw + 63) // 64])


KEYS = {11: ["lo_discount"], 50: ["lo_quantity"], 550: ["lo_quantity", "lo_discount"],
        3850: ["lo_quantity", "lo_discount", "d_year"]}
AGGS = {
    "all": [("sum", col("lo_revenue")), ("min", col("lo_revenue")), ("max", col("lo_supplycost")),
            ("avg", col("lo_revenue")), ("count", col("lo_revenue")), ("sum", col("lo_supplycost") - col("lo_revenue"))],
    "star": [("count", star()), ("max", col("lo_revenue")), ("min", col("lo_supplycost"))],
    "sum": [("sum", col("lo_supplycost"))],
}


def grouped(groups, aggs, nullable):
    b = PlanBuilder(datagen.ssb_tables(N, COLS), "LINEORDER", nullable=nullable, name=f"g{groups}")
    b.filter(col("lo_quantity").ne(7))
    b.join("DDATE", "lo_orderdate", where=col("d_month").le(9))
    return b.aggregate([queries._g(k) for k in KEYS[groups]], AGGS[aggs])


# 3,850 groups of six aggregates do not fit shared memory beside the row queues.
@pytest.mark.parametrize("groups,aggs", [(g, a) for g in sorted(KEYS) for a in sorted(AGGS) if (g, a) != (3850, "all")])
@pytest.mark.parametrize("kw", [dict(), dict(compact=1), dict(block_threads=128, group_merge=2),
                                dict(block_threads=256, items_per_thread=2, compact=2), dict(group_merge=1),
                                dict(stages=3, block_threads=512)], ids=str)
def test_group_words(loaded, groups, aggs, kw):
    check(loaded, grouped(groups, aggs, ("lo_revenue",)), make_tuning(group_placement=1, **kw))


@pytest.mark.parametrize("groups", [11, 550])
@pytest.mark.parametrize("kw", [dict(), dict(block_threads=128, items_per_thread=8)], ids=str)
def test_or_join_words(loaded, groups, kw):
    b = PlanBuilder(datagen.ssb_tables(N, COLS), "LINEORDER", nullable=("lo_revenue", "lo_commitdate"), name=f"o{groups}")
    b.filter(col("lo_quantity").lt(48))
    b.join("DDATE", ("lo_commitdate", "lo_orderdate"), where=col("d_year").ge(1993))
    check(loaded, b.aggregate([queries._g(k) for k in KEYS[groups]], AGGS["all"]), make_tuning(group_placement=1, **kw))


@pytest.mark.parametrize("kw", [dict(), dict(block_threads=128)], ids=str)
def test_multi_value_join_words(loaded, kw):
    b = PlanBuilder(datagen.ssb_tables(N, COLS), "LINEORDER", nullable=("lo_revenue",), name="m")
    b.join("DDATE", "lo_orderdate")
    b.join("PARTSUPP", "lo_partkey", where=col("ps_availqty").lt(5000))
    plan = b.aggregate([queries._g("d_year"), queries._g("ps_tier")],
                       [("count", star()), ("avg", col("lo_revenue")), ("min", col("ps_supplycost")),
                        ("sum", col("lo_revenue") * col("ps_availqty"))])
    check(loaded, plan, make_tuning(group_placement=1, **kw))
