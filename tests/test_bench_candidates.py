"""The benchmark's shared-scan candidates are programs of their own: none is compiled
and timed twice under two names."""
import random

import bench
from practice_b200 import _lib, queries
from practice_b200.engine import SHARED_DEFAULT, make_tuning


def test_distinct_programs():
    plans = [queries.template(t, random.Random(1)).text() for t in range(4)]
    programs = [_lib.shared_codegen(plans, make_tuning(**{**SHARED_DEFAULT, **c})) for c in bench.SHARED_CANDIDATES]
    assert len(set(programs)) == len(programs) == 5
