"""Scalar queries of the mask scan with more aggregates than a validity word has
bits: every SUM is valid once a row was added, none where no row passes."""
import numpy as np
import pytest

from practice_b200.engine import SHARED_DEFAULT, make_tuning
from practice_b200.plan import PlanBuilder, Table, col, lit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("naggs", [63, 64, 65, 129, 140])
@pytest.mark.parametrize("above", [500, 5000])
def test_every_sum_is_valid(naggs, above):
    from practice_b200.engine import Database
    rows = 3001
    rng = np.random.default_rng(naggs)
    cols = {"f_key": rng.integers(0, 1000, rows).astype(np.int32), "f_val": rng.integers(-99, 99, rows).astype(np.int32)}
    db = Database(0)
    for c, v in cols.items():
        db.load_column("F", c, v)
    db.set_rows("F", rows)
    b = PlanBuilder({"F": Table("F", list(cols), rows, fact=True)}, "F", name="mv")
    b.filter(col("f_key").ge(above))
    # (few distinct literals: a batch's parameters are bounded)
    plan = b.aggregate([], [("sum", col("f_val") if k else col("f_val") * lit(3)) for k in range(naggs)])
    got, = db.execute_shared([plan], make_tuning(**{**SHARED_DEFAULT, "cube": 0}))
    assert got.kernel_error == 0 and got.timing.mode == 0
    # (the oracle takes 32 aggregates)
    total = int(cols["f_val"][cols["f_key"] >= above].astype(np.int64).sum())
    assert got.words.view(np.int64).tolist() == [3 * total] + [total] * (naggs - 1)
    bits = np.unpackbits(got.validity.view(np.uint8), bitorder="little")[:naggs]
    assert bits.tolist() == [int(above < 1000)] * naggs
