"""Membership bits of a join in the fused scan, against the oracle, where the bit
after the window's last key starts a word, a 16-byte unit or nothing new: windows
around multiples of 32 and 128 keys, fact keys all inside, partly or all outside
the window, slots that hold another key's row, and row counts that end on a tile or within one."""
import numpy as np
import pytest

import oracle
from practice_b200.engine import make_tuning
from practice_b200.plan import Group, PlanBuilder, Table, col, star

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def db():
    from practice_b200.engine import Database
    return Database(0)


@pytest.mark.parametrize("length", [32, 96, 128, 127, 129, 256, 4096])
@pytest.mark.parametrize("keymin", [0, 1, -64])
@pytest.mark.parametrize("rows", [128, 4096 * 3, 4096 * 3 + 77])
@pytest.mark.parametrize("compact", [0, 1])
def test_bit_after_the_window(db, length, keymin, rows, compact):
    rng = np.random.default_rng(length * 31 + keymin + rows)
    inside = np.arange(keymin, keymin + length)
    # A third of the slots hold the key one window further on, a third none.
    keys = np.where(rng.random(length) < 0.5, inside, inside + length)[rng.random(length) < 0.67].astype(np.int32)
    attr = (np.abs(keys.astype(np.int64)) % 5).astype(np.int32)
    fkey = rng.integers(keymin, keymin + length, rows).astype(np.int32)
    out = rng.integers(keymin - 1, keymin + 2 * length + 2, rows).astype(np.int32)
    fkey = np.where(np.arange(rows) < rows // 2, fkey, out)  # first half: no key outside
    fkey[-3:] = [keymin + length - 1, keymin + length, keymin - 1]
    cols = {"f_key": fkey, "f_val": rng.integers(-100, 100, rows).astype(np.int32), "d_key": keys, "d_attr": attr}
    tabs = {"F": Table("F", ["f_key", "f_val"], rows, fact=True),
            "D": Table("D", ["d_key", "d_attr"], len(keys), key_col="d_key", key_min=keymin, key_max=keymin + length - 1)}
    db.reset()
    for t, names in (("F", ["f_key", "f_val"]), ("D", ["d_key", "d_attr"])):
        for c in names:
            db.load_column(t, c, cols[c])
        db.set_rows(t, len(cols[names[0]]))
    b = PlanBuilder(tabs, "F", name="bp")
    b.join("D", "f_key", where=col("d_attr").ne(3))
    plan = b.aggregate([Group(col("d_attr"), 0, 5, False)], [("count", star()), ("sum", col("f_val"))])
    ref = oracle.run_plan(plan.text(), cols, {}, {"F": rows, "D": len(keys)}, plan.group_slots * plan.storage_ts)
    got = db.execute(plan, make_tuning(compact=compact))
    assert got.kernel_error == 0
    np.testing.assert_array_equal(got.words, ref.words)
    np.testing.assert_array_equal(got.validity, ref.validity)
