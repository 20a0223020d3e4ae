"""Program texts that earlier generators wrote and a program has kept
(tests/golden/programs): cx_compile accepts them and they run as before.  v1 shared
programs bring their own staging, mask and aggregation warps, launch kinds and
memsets; the others build with a fixed block cap, or keep a spare bit behind their
bitmaps."""
import random
from pathlib import Path

import numpy as np
import pytest

import oracle
from practice_b200 import _lib, datagen, queries
from practice_b200.engine import SharedProgram, shape_key

TEXTS = Path(__file__).parent / "golden" / "programs"
N = 20_011
DIMS = ("DDATE", "CUSTOMER", "SUPPLIER", "PART", "PARTSUPP")


@pytest.mark.parametrize("name", sorted(p.stem for p in TEXTS.glob("*.txt")))
def test_compiles(name):
    _lib.Module((TEXTS / f"{name}.txt").read_text(), key="saved_" + name)


@pytest.fixture(scope="module")
def loaded():
    from practice_b200.engine import Database
    cols = sorted(set(queries.BATCH_COLS) | set(queries.Q31_COLS) | set(queries.MHT_COLS))
    ht = datagen.host_tables(3, N, cols, dims=DIMS)
    db = Database(0)
    db.load_host_tables(ht, datagen.ssb_tables(N, cols))
    return db, ht


def check(ht, plan, res, val):
    words = plan.group_slots * plan.storage_ts
    ref = oracle.run_plan(plan.text(), ht.columns, ht.validity, {"LINEORDER": N, **{d: datagen.DIM_ROWS[d] for d in DIMS}}, words)
    np.testing.assert_array_equal(res.cpu().numpy().view(np.uint64)[:words], ref.words)
    np.testing.assert_array_equal(val.cpu().numpy().view(np.uint64)[:(words + 63) // 64], ref.validity)


@pytest.mark.gpu
@pytest.mark.parametrize("name,plan", [("mht_v1", queries.mht_year_tier()), ("q31_spare_bit", queries.ssb_q31())])
def test_plain(loaded, name, plan):
    db, ht = loaded
    m = _lib.Module((TEXTS / f"{name}.txt").read_text(), key="saved_" + name)
    res, val = db.alloc_result(m)
    db.ctx.set_result(res.data_ptr(), res.numel(), val.data_ptr(), val.numel())
    db.ctx.execute(m, db.torch.cuda.current_stream().cuda_stream)
    db.ctx.sync()
    check(ht, plan, res, val)


@pytest.mark.gpu
@pytest.mark.parametrize("name", ["shared_v1", "shared_v2"])
@pytest.mark.parametrize("nq", [1, 33, 70])
@pytest.mark.parametrize("ranges", [True, False], ids=["cube", "masks"])
def test_shared(loaded, name, nq, ranges):
    db, ht = loaded
    m = _lib.Module((TEXTS / f"{name}.txt").read_text(), key="saved_" + name)
    rng = random.Random(nq)
    plans = [queries.template(1, rng) for _ in range(nq)]
    prog = SharedProgram(m, [shape_key(plans[0])], [len(_lib.plan_literals(plans[0].text()))])
    queries_, params, bufs = db.shared_prepare(prog, plans)
    # A year range of more than 65,536 values closes the cube path.
    db.ctx.set_column_range("d_d_year", 1992, 1998 if ranges else 1_000_000)
    db.ctx.shared_execute(m, queries_, params, db.torch.cuda.current_stream().cuda_stream)
    db.ctx.sync()
    assert db.ctx.timing().mode == (1 if ranges and name == "shared_v1" else 0)
    for p, (res, val, _) in zip(plans, bufs):
        check(ht, p, res, val)
