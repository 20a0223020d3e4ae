"""Hash tables built together with their membership bitmaps, against the oracle,
at the keys where the two can differ: key 0 and the window's first and last key,
keys outside the window whose slot is another key's, duplicate keys, windows that
are not a multiple of a bitmap word, one-row and empty dimensions, and fact keys
on both sides of the window."""
import numpy as np
import pytest

import oracle
from practice_b200.engine import make_tuning
from practice_b200.plan import Group, PlanBuilder, Table, col, star

pytestmark = pytest.mark.gpu

N = 20_011


def tables(keymin, length, rows):
    return {"F": Table("F", ["f_key", "f_val"], N, fact=True),
            "D": Table("D", ["d_key", "d_attr"], rows, key_col="d_key", key_min=keymin, key_max=keymin + length - 1)}


@pytest.fixture(scope="module")
def db():
    from practice_b200.engine import Database
    return Database(0)


@pytest.mark.parametrize("keymin,length", [(0, 1), (0, 31), (0, 33), (1, 64), (-5, 40), (-40, 40), (7, 1000), (-1000, 4099)])
@pytest.mark.parametrize("kind", ["window", "outside", "duplicates", "one", "empty"])
@pytest.mark.parametrize("payload", [False, True])
def test_build_and_bitmap(db, keymin, length, kind, payload):
    rng = np.random.default_rng(abs(keymin) * 7 + length)
    inside = np.arange(keymin, keymin + length)
    if kind == "window":
        keys = rng.permutation(inside)
    elif kind == "outside":
        # Keys past the window share slots with absent in-window ones: one key per slot.
        keys = np.where(rng.random(length) < 0.5, inside, inside + length)
    elif kind == "duplicates":
        keys = np.repeat(inside[::2], 2)
    else:
        keys = inside[:1] if kind == "one" else inside[:0]
    keys = keys.astype(np.int32)
    attr = (np.abs(keys.astype(np.int64) * 7) % 5).astype(np.int32)  # equal for equal keys
    fkey = rng.integers(keymin - length, keymin + 2 * length + 1, N).astype(np.int32)
    fkey[:3] = [0, keymin, keymin + length - 1]
    cols = {"f_key": fkey, "f_val": rng.integers(-100, 100, N).astype(np.int32), "d_key": keys, "d_attr": attr}
    tabs = tables(keymin, length, len(keys))
    db.reset()
    for t, names in (("F", ["f_key", "f_val"]), ("D", ["d_key", "d_attr"])):
        for c in names:
            db.load_column(t, c, cols[c])
        db.set_rows(t, len(cols[names[0]]))
    b = PlanBuilder(tabs, "F", name="bm")
    b.join("D", "f_key", where=col("d_attr").ne(3))
    if payload:
        plan = b.aggregate([Group(col("d_attr"), 0, 5, False)], [("count", star()), ("sum", col("f_val"))])
    else:
        plan = b.aggregate([], [("count", star()), ("sum", col("f_val"))])
    ref = oracle.run_plan(plan.text(), cols, {}, {"F": N, "D": len(keys)}, plan.group_slots * plan.storage_ts)
    for tuning in (None, make_tuning(bitmap_budget=0), make_tuning(compact=1, block_threads=256)):
        got = db.execute(plan, tuning)
        assert got.kernel_error == 0
        np.testing.assert_array_equal(got.words, ref.words)
        np.testing.assert_array_equal(got.validity, ref.validity)
