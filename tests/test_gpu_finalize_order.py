"""ORDER BY of cx_finalize on group tables made directly: sizes at the edges of
its sorted runs (1024 groups), of one ranking pass (65,536 groups) and past it,
NULL keys, DESC, INT64 / UINT64 / FLOAT64 keys with infinities and both zeros,
and NaN keys, whose order is the comparator's under a bitonic network
(src/core/visitor.cpp:307-358 compares; a NaN is equal to everything).  Whole
words are compared, so every result has to be equal bit for bit."""
import functools
import struct

import numpy as np
import pytest

from practice_b200 import _lib

pytestmark = pytest.mark.gpu

INT, UINT, DBL = _lib.COL_INT64, _lib.COL_UINT64, _lib.COL_FLOAT64


def table(groups, density, kinds, seed, nan=False):
    """Group tuples: one column per kind, few distinct values so that ties reach the later keys."""
    rng = np.random.default_rng(seed)
    cols = []
    for k in kinds:
        if k == DBL:
            pool = np.array([0.0, -0.0, 1.5, -2.5, np.inf, -np.inf, 1e300, 5e-324] + ([np.nan] * 3 if nan else []))
            cols.append(rng.choice(pool, groups).view(np.uint64))
        elif k == INT:
            cols.append(rng.integers(-5, 6, groups).astype(np.int64).view(np.uint64))
        else:
            cols.append(rng.choice(np.array([1, 2, 1 << 31, 1 << 63, (1 << 64) - 1], dtype=np.uint64), groups))
    words = np.stack(cols, axis=1)
    present = rng.random(groups) < density
    bits = rng.random((groups, len(kinds))) < 0.8
    words[~present] = 0
    bits[~present] = False
    return words, bits


def value(kind, x):
    x = int(x)
    if kind == INT:
        return x - (1 << 64) if x >> 63 else x
    return struct.unpack("<d", struct.pack("<Q", x))[0] if kind == DBL else x


def expected(words, bits, kinds, nullable, keys, limit, network=False):
    rows = [g for g in range(len(words)) if bits[g].any() or words[g].any()]
    vals = {g: [(bool(bits[g][c]) or not nullable[c], value(kinds[c], words[g][c])) for c, _ in keys] for g in rows}
    place = {g: i for i, g in enumerate(rows)}

    def cmp(l, r):
        for (c, desc), (lv, a), (rv, b) in zip(keys, vals[l], vals[r]):
            if lv != rv:
                return -1 if lv else 1
            if not lv:
                continue
            if b < a:
                return -1 if desc else 1
            if a < b:
                return 1 if desc else -1
        return place[l] - place[r]

    if network:
        n = 1
        while n < len(rows):
            n <<= 1
        s = rows + [None] * (n - len(rows))
        k = 2
        while k <= n:
            j = k >> 1
            while j:
                for i in range(n):
                    x = i ^ j
                    if x > i:
                        l, r = s[i], s[x]
                        rb = r is not None and (l is None or cmp(l, r) > 0)
                        lb = l is not r and not rb
                        if rb if not i & k else lb:
                            s[i], s[x] = r, l
                j >>= 1
            k <<= 1
        rows = s[:len(rows)]
    else:
        rows = sorted(rows, key=functools.cmp_to_key(cmp))
    return rows if limit is None else rows[:limit]


def run(words, bits, kinds, nullable, keys, limit):
    import torch
    groups, nc = words.shape
    flat = np.zeros((groups * nc + 63) // 64 * 64, dtype=np.uint8)
    flat[:groups * nc] = bits.reshape(-1)
    val = torch.from_numpy(np.packbits(flat, bitorder="little").view(np.int64)).cuda()
    src = torch.from_numpy(words.reshape(-1).view(np.int64).copy()).cuda()
    cols = torch.full((nc * groups,), -7, dtype=torch.int64, device="cuda")
    vw = (groups + 63) // 64
    cval = torch.full((nc * vw,), -1, dtype=torch.int64, device="cuda")
    n = _lib.finalize(src.data_ptr(), val.data_ptr(), groups, nc, kinds, nullable, False, False, keys, limit,
                      cols.data_ptr(), cval.data_ptr(), groups, torch.cuda.current_stream().cuda_stream)
    v = np.unpackbits(cval.cpu().numpy().view(np.uint8), bitorder="little").reshape(nc, -1)
    return n, cols.cpu().numpy().view(np.uint64).reshape(nc, groups), v


def check(words, bits, kinds, nullable, keys, limit, network=False):
    want = expected(words, bits, kinds, nullable, keys, limit, network)
    n, cols, v = run(words, bits, kinds, nullable, keys, limit)
    assert n == len(want)
    for c in range(len(kinds)):
        np.testing.assert_array_equal(cols[c, :n], words[want, c])
        np.testing.assert_array_equal(v[c, :n], [1 if bits[g][c] or not nullable[c] else 0 for g in want])
        assert not v[c, n:].any()


@pytest.mark.parametrize("groups,density", [(1, 1.0), (2, 1.0), (63, 1.0), (64, 0.5), (1023, 1.0), (1024, 1.0), (1025, 1.0),
                                            (2049, 0.02), (5000, 0.9), (65_536, 0.3), (65_537, 0.3), (70_001, 1.0)])
def test_order_by_integers(groups, density):
    words, bits = table(groups, density, [INT, UINT, INT], groups)
    keys = [(0, False), (1, True), (2, False)]
    check(words, bits, [INT, UINT, INT], [True, False, True], keys, None)
    check(words, bits, [INT, UINT, INT], [False, False, False], [(1, True)], min(7, groups))


@pytest.mark.parametrize("groups", [1, 1024, 1025, 40_000])
@pytest.mark.parametrize("desc", [False, True])
def test_order_by_doubles(groups, desc):
    words, bits = table(groups, 0.9, [DBL, INT], groups + desc)
    check(words, bits, [DBL, INT], [True, True], [(0, desc), (1, not desc)], None)


def test_order_by_doubles_with_nan_keeps_the_network_order():
    words, bits = table(300, 0.9, [DBL, INT], 5, nan=True)
    check(words, bits, [DBL, INT], [True, False], [(0, True), (1, False)], None, network=True)
    check(words, bits, [DBL, INT], [True, False], [(0, False)], 11, network=True)


@pytest.mark.parametrize("groups", [1, 2048, 2049, 70_001])
@pytest.mark.parametrize("limit", [None, 0, 1, 64, 65])
def test_limit_without_order(groups, limit):
    words, bits = table(groups, 0.7, [INT, UINT], groups)
    check(words, bits, [INT, UINT], [True, False], [], limit)


def test_most_sort_words():
    """Eight nullable keys: sixteen sort words per row."""
    kinds = [INT] * 8
    words, bits = table(3000, 0.9, kinds, 9)
    words[:, :6] &= np.uint64(1)
    check(words, bits, kinds, [True] * 8, [(c, c % 2 == 1) for c in range(8)], None)
