"""A membership bitmap takes exactly a bit per slot of its window, to 16 bytes: one
that fills the budget takes the budget, and a launch shape whose shared memory is
filled to the last byte by it is accepted."""
import re

import pytest

from practice_b200 import _lib
from practice_b200.engine import make_tuning
from practice_b200.plan import PlanBuilder, Table, star


def scan_smem(length, **kw):
    tabs = {"F": Table("F", ["f_key"], 1000, fact=True),
            "D": Table("D", ["d_key"], length, key_col="d_key", key_min=1, key_max=length)}
    b = PlanBuilder(tabs, "F", name="bb")
    b.join("D", "f_key")
    src = _lib.codegen(b.aggregate([], [("count", star())]).text(), make_tuning(block_threads=1024, items_per_thread=4, **kw))
    return int(re.search(r"^kernel \S+ scan 0 \d+ \d+ (\d+) ", src, re.M).group(1))


@pytest.mark.parametrize("length", [1, 31, 32, 33, 127, 128, 129, 256, 4096, 393_216])
def test_bytes(length):
    budget = ((length + 31) // 32 * 4 + 15) // 16 * 16
    none = scan_smem(length, bitmap_budget=0)
    assert none == 512  # barriers and reduction words; the sum is rounded to 128 bytes
    assert scan_smem(length, bitmap_budget=budget) == (none + budget + 127) // 128 * 128
    assert scan_smem(length, bitmap_budget=budget - 1) == none


def test_full_shared_memory():
    # Eleven stages of one column, their barriers and 48 KiB of bitmap: 227 KiB.
    assert scan_smem(393_216, stages=11, bitmap_budget=49_152) == 227 * 1024
