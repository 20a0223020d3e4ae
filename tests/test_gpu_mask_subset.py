"""Mask-scan passes that read some of their program's columns (a batch of some of
its shapes, and a batch cut into passes by shape): full tiles are read with vector
loads of just those columns; results against the oracle, each query alone."""
import random

import numpy as np
import pytest

import oracle
from practice_b200 import _lib, datagen, queries
from practice_b200.engine import SHARED_DEFAULT, make_tuning

COLS = sorted(queries.BATCH_COLS)
TUNING = {**SHARED_DEFAULT, "cube": 0}


def mix(n, rng, count=8, kinds=range(4)):
    kinds = list(kinds)
    return [queries.template(kinds[i % len(kinds)], rng, n) for i in range(count)]


def test_vector_loads_of_a_subset():
    src = _lib.shared_codegen([p.text() for p in mix(1000, random.Random(1), 4)], make_tuning(**TUNING))
    scan = src[src.index("SharedScan_LINEORDER(const"):]
    for k in range(len(COLS)):
        assert f"if ((m_cols >> {k}) & 1ULL) WarpLoadTileV<IPT>(" in scan


@pytest.fixture(scope="module")
def db():
    from practice_b200.engine import Database
    return Database(0)


def check(db, ht, plans, bufs):
    rows = {"LINEORDER": ht.fact_rows, **{d: datagen.DIM_ROWS[d] for d in ("DDATE", "CUSTOMER", "SUPPLIER", "PART")}}
    for p, (res, val, words) in zip(plans, bufs):
        ref = oracle.run_plan(p.text(), ht.columns, ht.validity, rows, p.group_slots * p.storage_ts)
        np.testing.assert_array_equal(res.cpu().numpy().view(np.uint64)[:words], ref.words, err_msg=p.name)
        np.testing.assert_array_equal(val.cpu().numpy().view(np.uint64)[:(words + 63) // 64], ref.validity, err_msg=p.name)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [64, 2048, 40_031])
@pytest.mark.parametrize("kinds", [(0,), (1,), (2,), (3,), (0, 3), (1, 2, 3)])
@pytest.mark.parametrize("row0", [0, 2, 3])
def test_some_shapes(db, n, kinds, row0):
    ht = datagen.host_tables(11, n, COLS)
    db.reset()
    db.load_host_tables(ht, datagen.ssb_tables(n, COLS))
    rng = random.Random(n)
    prog = db.shared_program(mix(n, rng, 4), make_tuning(**TUNING))
    plans = mix(n, rng, 9, kinds)
    queries_, params, bufs = db.shared_prepare(prog, plans)
    stream = db.torch.cuda.current_stream().cuda_stream
    at = 0
    for size in ([row0] if row0 else []) + [n]:  # a second range from an even or odd row on
        db.ctx.shared_execute_rows(prog.module, queries_, params, at, size, [at > 0] * len(plans), stream)
        db.ctx.sync()
        at += size
    check(db, ht, plans, bufs)


@pytest.mark.gpu
def test_passes_by_shape(db):
    n = 40_031
    ht = datagen.host_tables(12, n, COLS)
    db.reset()
    db.load_host_tables(ht, datagen.ssb_tables(n, COLS))
    plans = mix(n, random.Random(5), 130)
    prog = db.shared_program(plans, make_tuning(**TUNING))
    queries_, params, bufs = db.shared_prepare(prog, plans)
    db.ctx.shared_execute(prog.module, queries_, params, db.torch.cuda.current_stream().cuda_stream)
    db.ctx.sync()
    check(db, ht, plans, bufs)
