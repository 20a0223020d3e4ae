"""COUNT past 2^32 rows of one CTA.  The scans count rows per CTA in 32-bit words of
shared memory; one SM with one CTA and 4.3 billion rows (2.1 billion where an
OR-join counts each twice) passes such a word.  Exactly 2^32 rows of one group would
leave 0, which also stands for a group without rows; the last row is another
group's, the only one with a valid value, and is read from a later launch's
validity words.  One 17 GB column serves as every column."""
import numpy as np
import pytest

from practice_b200 import _lib
from practice_b200.engine import make_tuning
from practice_b200.plan import Group, PlanBuilder, Table, col, star

pytestmark = pytest.mark.gpu

WRAP = 1 << 32


@pytest.fixture(scope="module")
def db():
    from practice_b200.engine import Database
    db = Database(0)
    yield db
    db.reset()
    db.torch.cuda.empty_cache()


def load(db, n, names, value=0, last=999):
    """Columns `names` over one tensor: `value`, and `last` in the last row."""
    db.reset()
    _lib.check(_lib.lib.cx_ctx_set_sm_count(db.ctx.handle, 1), "cx_ctx_set_sm_count")
    t = db.torch.full((n,), value, dtype=db.torch.int32, device=db.device)
    t[-1] = last
    for c in names:
        db.load_column("F", c, t)
    db.set_rows("F", n)


def last_row_valid(db, n, name):
    words = db.torch.zeros((n + 63) // 64, dtype=db.torch.int64, device=db.device)
    words[-1] = -(1 << 63) if n % 64 == 0 else 1 << ((n - 1) % 64)
    db.load_validity(name, words)


def rows_of(got, plan):
    """The present groups' tuples and validity bits by their key (a sparse result has no bits)."""
    words = got.words.view(np.int64).reshape(plan.group_slots, plan.storage_ts)
    bits = np.unpackbits(got.validity.view(np.uint8), bitorder="little")[: words.size].reshape(words.shape)
    if plan.sparse:
        return {int(w[0]): (w.tolist(), [1] * len(w)) for w in words if w.any()}
    return {int(words[g][0]): (words[g].tolist(), bits[g].tolist()) for g in range(plan.group_slots) if bits[g][0]}


def test_plain_scan(db):
    n = WRAP + 1
    load(db, n, ["f_key", "f_val"])
    last_row_valid(db, n, "f_val")
    b = PlanBuilder({"F": Table("F", ["f_key", "f_val"], n, fact=True)}, "F", nullable=("f_val",), name="count_plain")
    # (a SUM beside the COUNT: one copy of each word in shared memory)
    plan = b.aggregate([Group(col("f_key"), 0, 1000, False)], [("count", star()), ("sum", col("f_val"))])
    got = db.execute(plan, make_tuning(ctas_per_sm=1))
    assert got.kernel_error == 0 and got.timing.scan_grid == 1
    assert rows_of(got, plan) == {0: ([0, WRAP, 0], [1, 1, 0]), 999: ([999, 1, 999], [1, 1, 1])}


def test_or_join(db):
    n = WRAP // 2 + 1
    load(db, n, ["f_a"], value=1, last=3)
    t = db.torch.full((n,), 2, dtype=db.torch.int32, device=db.device)
    t[-1] = 4
    db.load_column("F", "f_b", t)
    db.load_column("F", "f_val", t)
    last_row_valid(db, n, "f_val")
    dim = np.arange(1, 5, dtype=np.int32)
    db.load_column("D", "d_key", dim)
    db.load_column("D", "d_attr", np.where(dim <= 2, 0, 999).astype(np.int32))
    db.set_rows("D", 4)
    tabs = {"F": Table("F", ["f_a", "f_b", "f_val"], n, fact=True),
            "D": Table("D", ["d_key", "d_attr"], 4, key_col="d_key", key_min=1, key_max=4)}
    b = PlanBuilder(tabs, "F", nullable=("f_val",), name="count_or")
    b.join("D", ("f_a", "f_b"))
    plan = b.aggregate([Group(col("d_attr"), 0, 1000, False)], [("count", star()), ("sum", col("f_val"))])
    got = db.execute(plan, make_tuning(ctas_per_sm=1))
    assert got.kernel_error == 0 and got.timing.scan_grid == 1
    assert rows_of(got, plan) == {0: ([0, WRAP, 0], [1, 1, 0]), 999: ([999, 2, 8], [1, 1, 1])}


@pytest.mark.parametrize("cube", [0, 4], ids=["masks", "cube"])
def test_shared_scan(db, cube):
    n = WRAP + 1
    load(db, n, ["f_key"])
    b = PlanBuilder({"F": Table("F", ["f_key"], n, fact=True)}, "F", name="count_shared")
    plan = b.aggregate([Group(col("f_key"), 0, 1000, False)], [("count", star())])
    got, = db.execute_shared([plan], make_tuning(block_threads=1024, items_per_thread=1, stages=3, ctas_per_sm=1, cube=cube))
    assert got.kernel_error == 0 and got.timing.scan_grid == 1 and got.timing.mode == (1 if cube else 0)
    assert rows_of(got, plan) == {0: ([0, WRAP], [1, 1]), 999: ([999, 1], [1, 1])}
