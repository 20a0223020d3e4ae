"""Mask scan: the tables of a full pass of 64 queries fit the shared memory that the
host gives them, whatever the copies of their words, wherever one copy of each does."""
import re

import pytest

from practice_b200 import _lib
from practice_b200.engine import SHARED_DEFAULT, make_tuning
from practice_b200.plan import Group, PlanBuilder, Table, col, star

F = Table("F", ["f_key", "f_val"], 1000, fact=True)


@pytest.mark.parametrize("card", [1, 7, 10, 12, 31, 64, 100, 128])
@pytest.mark.parametrize("aggs", [[("sum", "f_val")], [("sum", "f_val"), ("count", None)], [("count", None)]], ids=str)
@pytest.mark.parametrize("block,ctas", [(1024, 1), (1024, 2), (512, 1), (512, 2), (256, 4)])
def test_a_full_pass_fits(card, aggs, block, ctas):
    b = PlanBuilder({"F": F}, "F", name="qt")
    plan = b.aggregate([Group(col("f_key"), 0, card, False)], [(fn, col(c) if c else star()) for fn, c in aggs])
    src = _lib.shared_codegen([plan.text()], make_tuning(**{**SHARED_DEFAULT, "block_threads": block, "ctas_per_sm": ctas, "cube": 0}))
    sshape = re.search(r"^sshape 0 (.*)$", src, re.M).group(1).split()
    tab, bits = int(sshape[-2]) * 8, int(sshape[-1]) * 4
    smem = int(re.search(r"^kernel \S+ sharedscan 0 \d+ \d+ (\d+) ", src, re.M).group(1))
    one = card * sum(4 if fn == "count" else 8 for fn, _ in aggs)
    resident = min(ctas, 1024 // block)
    cap = min(200 * 1024, 233472 // resident - 1024)
    assert tab >= one
    if smem + 64 * (one + bits + 8) + 64 <= cap:
        assert smem + 64 * (tab + bits) + 64 <= cap
