"""Mask scan over group domains that a query's shared-memory table does not hold
whole: some groups lie in it, the others go to the result.  Domains just above the
limit and far above, few live groups and all of them, one and two mask words of
queries, values of both signs, COUNT and SUM, a value that holds a literal;
whole results against the oracle."""
import re

import numpy as np
import pytest

import oracle
from practice_b200 import _lib
from practice_b200.engine import SHARED_DEFAULT, make_tuning
from practice_b200.plan import Group, PlanBuilder, Table, col, lit, star

ROWS = 30_011


def plans(nq, card, live, aggs, literal):
    t = {"F": Table("F", ["f_key", "f_val"], ROWS, fact=True)}
    out = []
    for q in range(nq):
        b = PlanBuilder(t, "F", name="wd")
        b.filter(col("f_val").ge(-100 + q))
        val = col("f_val") * lit(1 + q % 3) if literal else col("f_val")
        out.append(b.aggregate([Group(col("f_key"), 0, card, False)],
                               [("sum", val) if a == "sum" else ("count", star()) for a in aggs]))
    return out


TUNING = {**SHARED_DEFAULT, "cube": 0}


@pytest.mark.parametrize("card,aggs", [(513, ["sum"]), (1025, ["count"]), (5000, ["sum", "count"]), (70_000, ["sum"])])
def test_wide_domains_have_a_table(card, aggs):
    src = _lib.shared_codegen([plans(1, card, card, aggs, False)[0].text()], make_tuning(**TUNING))
    sshape = re.search(r"^sshape 0 (.*)$", src, re.M).group(1).split()
    assert int(sshape[-2]) > 0


@pytest.mark.gpu
@pytest.mark.parametrize("nq", [1, 8, 33, 64])
@pytest.mark.parametrize("card,aggs", [(513, ["sum"]), (1025, ["count"]), (5000, ["sum", "count"]), (70_000, ["count", "sum"])])
@pytest.mark.parametrize("live", [1, 11, 300, 513])
@pytest.mark.parametrize("literal", [False, True])
def test_against_the_oracle(nq, card, aggs, live, literal):
    from practice_b200.engine import Database
    rng = np.random.default_rng(card + live)
    step = max(1, (card - 3) // live)
    key = (rng.integers(0, live, ROWS) * step).clip(0, card - 3)
    cols = {"f_key": key.astype(np.int32), "f_val": rng.integers(-100, 100, ROWS).astype(np.int32)}
    db = Database(0)
    for c, v in cols.items():
        db.load_column("F", c, v)
    db.set_rows("F", ROWS)
    batch = plans(nq, card, live, aggs, literal)
    for p, got in zip(batch, db.execute_shared(batch, make_tuning(**TUNING))):
        ref = oracle.run_plan(p.text(), cols, {}, {"F": ROWS}, p.group_slots * p.storage_ts)
        assert got.kernel_error == 0 and got.timing.mode == 0
        np.testing.assert_array_equal(got.words, ref.words)
        np.testing.assert_array_equal(got.validity, ref.validity)
