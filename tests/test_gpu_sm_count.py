"""cx_ctx_set_sm_count sizes the build grids too: each table's part takes its blocks
from the arguments, so that the kernel and the launch agree whatever the count.
With one SM a part has 16 blocks for tables of up to 300,000 rows, each of several
tiles; results against the oracle."""
import random
import re

import numpy as np
import pytest

import oracle
from practice_b200 import _lib, datagen, queries
from practice_b200.engine import SHARED_DEFAULT, make_tuning

N = 20_011
COLS = sorted(set(queries.BATCH_COLS) | set(queries.MHT_COLS))


def test_no_fixed_cap():
    plan = queries.ssb_q31(N)
    for src, kernel in ((_lib.codegen(plan.text()), "build_tables"),
                        (_lib.shared_codegen([plan.text()], make_tuning(**SHARED_DEFAULT)), "index_tables")):
        assert re.search(rf"^kernel {kernel} builds 0 \d+ \d+ 0 3 ", src, re.M)
        body = src[src.index(f" {kernel}(const CxArgs a)"):]
        assert body[: body.index("\n}")].count("a.build_cap") == 3


@pytest.mark.gpu
@pytest.mark.parametrize("sms", [1, 3, 148])
@pytest.mark.parametrize("what", ["plain", "mht", "masks", "cube"])
def test_against_the_oracle(sms, what):
    from practice_b200.engine import Database
    ht = datagen.host_tables(5, N, COLS, dims=("DDATE", "CUSTOMER", "SUPPLIER", "PART", "PARTSUPP"))
    db = Database(0)
    db.load_host_tables(ht, datagen.ssb_tables(N, COLS))
    _lib.check(_lib.lib.cx_ctx_set_sm_count(db.ctx.handle, sms), "cx_ctx_set_sm_count")
    rows = {"LINEORDER": N, **{d: datagen.DIM_ROWS[d] for d in ("DDATE", "CUSTOMER", "SUPPLIER", "PART", "PARTSUPP")}}
    if what in ("plain", "mht"):
        plans = [queries.ssb_q31(N)] if what == "plain" else [queries.mht_brand(N)]
        got = [db.execute(p) for p in plans]
    else:
        rng = random.Random(sms)
        plans = [queries.template(t, rng, N) for t in range(4)]
        got = db.execute_shared(plans, make_tuning(**{**SHARED_DEFAULT, **({"cube": 0} if what == "masks" else {})}))
    for p, g in zip(plans, got):
        ref = oracle.run_plan(p.text(), ht.columns, ht.validity, rows, p.group_slots * p.storage_ts)
        assert g.kernel_error == 0
        np.testing.assert_array_equal(g.words, ref.words, err_msg=p.name)
        np.testing.assert_array_equal(g.validity, ref.validity, err_msg=p.name)
