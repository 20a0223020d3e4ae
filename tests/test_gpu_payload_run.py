"""Payloads of neighbouring joins fetched together, against the oracle: two and
three joins in a row, a join without a payload or a filter between them, keys
outside a window, and row counts on and off a tile."""
import numpy as np
import pytest

import oracle
from practice_b200.engine import make_tuning
from practice_b200.plan import Group, PlanBuilder, Table, col, star

pytestmark = pytest.mark.gpu

DIMS = {"A": ("a", 0, 40), "B": ("b", 7, 128), "C": ("c", -5, 300)}


@pytest.fixture(scope="module")
def db():
    from practice_b200.engine import Database
    return Database(0)


@pytest.mark.parametrize("rows", [1, 128, 128 * 33 + 31])
@pytest.mark.parametrize("form", ["two", "three", "bare", "filter"])
@pytest.mark.parametrize("compact", [0, 1])
def test_fetched_together(db, rows, form, compact):
    rng = np.random.default_rng(rows + len(form))
    fcols = ["f_a", "f_b", "f_c", "f_val"]
    tabs = {"F": Table("F", fcols, rows, fact=True)}
    cols = {"f_val": rng.integers(-100, 100, rows).astype(np.int32)}
    for name, (x, kmin, length) in DIMS.items():
        keys = np.arange(kmin, kmin + length)
        # Some slots hold the key one window further on.
        keys = np.where(rng.random(length) < 0.3, keys + length, keys).astype(np.int32)
        tabs[name] = Table(name, [f"{x}_key", f"{x}_attr"], length, key_col=f"{x}_key", key_min=kmin, key_max=kmin + length - 1)
        cols[f"{x}_key"], cols[f"{x}_attr"] = keys, rng.integers(0, 5, length).astype(np.int32)
        cols[f"f_{x}"] = rng.integers(kmin, kmin + 2 * length, rows).astype(np.int32)
    db.reset()
    for t, tab in tabs.items():
        names = fcols if t == "F" else [f"{DIMS[t][0]}_key", f"{DIMS[t][0]}_attr"]
        for c in names:
            db.load_column(t, c, cols[c])
        db.set_rows(t, len(cols[names[0]]))
    b = PlanBuilder(tabs, "F", name="pr")
    b.join("A", "f_a")
    if form == "filter":
        b.filter(col("a_attr").ne(1))
    b.join("B", "f_b", where=col("b_attr").ne(3))
    if form != "two":
        b.join("C", "f_c")
    groups = [Group(col(f"{x}_attr"), 0, 5, False) for x in ("ab" if form in ("two", "bare") else "abc")]
    plan = b.aggregate(groups, [("count", star()), ("sum", col("f_val"))])
    ref = oracle.run_plan(plan.text(), cols, {}, {t: len(cols[f"{DIMS[t][0]}_key"]) if t != "F" else rows for t in tabs},
                          plan.group_slots * plan.storage_ts)
    got = db.execute(plan, make_tuning(compact=compact))
    assert got.kernel_error == 0
    np.testing.assert_array_equal(got.words, ref.words)
    np.testing.assert_array_equal(got.validity, ref.validity)
