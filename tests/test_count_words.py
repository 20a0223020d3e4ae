"""The launch plan states how often one fact row can add to a 32-bit count of a
CTA: the host bounds the rows of a launch by it.  0 where counts are 64 bits."""
import re

import pytest

from practice_b200 import _lib, queries
from practice_b200.engine import SHARED_DEFAULT, make_tuning
from practice_b200.plan import Group, PlanBuilder, Table, col, star

F = Table("F", ["f_key", "f_b", "f_c"], 1000, fact=True)
DIMS = [Table(d, [f"{d.lower()}_key", f"{d.lower()}_attr"], 9, key_col=f"{d.lower()}_key", key_min=1, key_max=9) for d in ("D", "E")]


def plan(joins=(), aggs=(("count", star()),)):
    b = PlanBuilder({t.name: t for t in [F, *DIMS]}, "F", name="cw")
    for d, keys in joins:
        b.join(d, keys)
    return b.aggregate([Group(col("f_key"), 0, 1000, False)], list(aggs))


def rowmax(src):
    return int(re.search(r"^rowmax (\d+)$", src, re.M).group(1))


@pytest.mark.parametrize("p,want", [
    (plan(), 1),
    (plan(aggs=[("avg", col("f_b"))]), 1),
    (plan(aggs=[("sum", col("f_b")), ("min", col("f_b"))]), 0),
    (plan([("D", ("f_key", "f_b", "f_c"))]), 3),
    (plan([("D", ("f_key", "f_b", "f_c")), ("E", ("f_b", "f_c"))]), 6),
    (queries.mht_brand(1000), 0),         # global 64-bit words
    (queries.mht_year_tier(1000), 0),     # two words a count
    (queries.kat_plans()["q1"], 0),       # scalar: registers
])
def test_plain(p, want):
    assert rowmax(_lib.codegen(p.text())) == want


def test_global_tables_and_64_bit_tables():
    assert rowmax(_lib.codegen(plan().text(), make_tuning(group_placement=2))) == 0
    assert rowmax(_lib.codegen(plan().text(), make_tuning(group_merge=1))) == 0


def test_shared():
    t = make_tuning(**SHARED_DEFAULT)
    assert rowmax(_lib.shared_codegen([plan().text()], t)) == 1
    assert rowmax(_lib.shared_codegen([plan(aggs=[("sum", col("f_b"))]).text()], t)) == 0


@pytest.mark.parametrize("bad", ["-1", "65537"])
def test_reader_refuses(bad):
    src = re.sub(r"^rowmax \d+$", f"rowmax {bad}", _lib.codegen(plan().text()), flags=re.M)
    with pytest.raises(_lib.CxError):
        _lib.Module(src, key="cw")
