"""Sparse compaction (CompactSparseAggregateResult, src/db/database_instance.cpp:286-307)
at the edges of its blocks of 2048 groups and of the self-summed block counts
(2048 blocks), for tuples of one word and more, tables that are not 16-byte
aligned, and empty and full results; both entry points against numpy."""
import numpy as np
import pytest

from practice_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("groups", [1, 31, 2047, 2048, 2049, 100_003, 2048 * 2048, 2048 * 2048 + 1])
@pytest.mark.parametrize("ts,shift", [(1, 0), (2, 1), (5, 0), (5, 1), (7, 0)])
@pytest.mark.parametrize("density", [0.0, 0.01, 1.0])
def test_compaction_matches_numpy(groups, ts, shift, density):
    import torch
    rng = np.random.default_rng(groups * 31 + ts)
    # One non-zero word at a random place of each present tuple.
    words = np.zeros((groups, ts), dtype=np.int64)
    rows = np.flatnonzero(rng.random(groups) < density)
    words[rows, rng.integers(0, ts, len(rows))] = rng.integers(1, 1 << 62, len(rows))
    buf = torch.zeros(groups * ts + shift, dtype=torch.int64, device="cuda")
    src = buf[shift:]
    src.copy_(torch.from_numpy(words.reshape(-1)))
    for fn in (_lib.lib.cx_compact_sparse, _lib.lib.cx_compact_sparse_noalloc):
        dst = torch.full((len(rows) * ts + 1,), -3, dtype=torch.int64, device="cuda")
        cnt = torch.full((1,), -1, dtype=torch.int64, device="cuda")
        _lib.check(fn(src.data_ptr(), groups, ts, dst.data_ptr(), cnt.data_ptr(),
                      torch.cuda.current_stream().cuda_stream))
        assert int(cnt.item()) == len(rows)
        got = dst.cpu().numpy()
        np.testing.assert_array_equal(got[:-1], words[rows].reshape(-1))
        assert got[-1] == -3
