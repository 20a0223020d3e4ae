"""Presence bits of cubes without COUNT, against the oracle, where the host places
them differently: in shared memory (four templates: 175,000 cells, 22 KB of bits
beside dimension words of one byte), beside a gathered dimension that keeps its L1
(a fifth shape makes a date word two bytes, 122 KB, too many for shared memory), in
the cube itself (4.8 million cells, 600 KB), and for cubes that lie in shared
memory.  SUMs that are 0, and cells whose first rows add 0, count as present."""
import random

import numpy as np
import pytest

import oracle
from practice_b200 import datagen, queries
from practice_b200.engine import SHARED_DEFAULT, make_tuning
from practice_b200.plan import PlanBuilder, and_, col

pytestmark = pytest.mark.gpu

COLS = sorted(queries.BATCH_COLS)
DIMS = ("DDATE", "CUSTOMER", "SUPPLIER", "PART")


def wide(rng, n):
    b = PlanBuilder(datagen.ssb_tables(n, COLS), "LINEORDER", name="wide")
    d = rng.randint(0, 8)
    b.filter(and_(col("lo_discount").ge(d), col("lo_discount").le(d + 2)))
    b.join("CUSTOMER", "lo_custkey")
    b.join("SUPPLIER", "lo_suppkey")
    b.join("DDATE", "lo_orderdate", where=col("d_year").ge(rng.randint(1992, 1998)))
    return b.aggregate([queries._g("c_city"), queries._g("s_city")], [("sum", col("lo_revenue"))])


def batch(kind, n):
    rng = random.Random(n)
    plans = [queries.template(t, rng, n) for t in range(4) for _ in range(2)]
    if kind == "gathered":
        plans += [queries.city_pairs(rng, n) for _ in range(2)]
    elif kind == "own":
        plans = plans[:2] + [wide(rng, n) for _ in range(2)]
    elif kind == "shared":
        plans = plans[:6]
    return plans


@pytest.fixture(scope="module")
def db():
    from practice_b200.engine import Database
    return Database(0)


@pytest.mark.parametrize("kind", ["bits", "gathered", "own", "shared"])
@pytest.mark.parametrize("n", [1, 127, 60_011])
@pytest.mark.parametrize("zero", [False, True])
def test_placements(db, kind, n, zero):
    ht = datagen.host_tables(23, n, COLS)
    if zero:  # every sum 0: revenue and supply cost alike, the discount 0
        ht.columns["lo_revenue"] = np.where(np.arange(n) % 3 == 0, 0, ht.columns["lo_supplycost"]).astype(np.int32)
        ht.columns["lo_revenue"][: n // 2] = 0
        ht.columns["lo_supplycost"] = ht.columns["lo_revenue"].copy()
    db.reset()
    db.load_host_tables(ht, datagen.ssb_tables(n, COLS))
    rows = {"LINEORDER": n, **{d: datagen.DIM_ROWS[d] for d in DIMS}}
    plans = batch(kind, n)
    for p, got in zip(plans, db.execute_shared(plans, make_tuning(**SHARED_DEFAULT))):
        ref = oracle.run_plan(p.text(), ht.columns, ht.validity, rows, p.group_slots * p.storage_ts)
        assert got.kernel_error == 0 and got.timing.mode == 1
        np.testing.assert_array_equal(got.words, ref.words, err_msg=p.name)
        np.testing.assert_array_equal(got.validity, ref.validity, err_msg=p.name)
