"""cx_finalize from several streams and threads at once: their scratch comes from one
pool per device, in stream order.  Every thread orders its own buffer by its own
keys on its own stream, on the path without a row count and on the one with (a
table above 65,536 groups), and compares each call with the first one alone."""
import threading

import numpy as np
import pytest
import torch

from practice_b200 import _lib

pytestmark = pytest.mark.gpu

INT64, UINT64 = 0, 1


def finalize(src, groups, keys, limit, out, vout, stream):
    cap = max(groups, 1)
    n = _lib.finalize(src.data_ptr(), 0, groups, 2, [UINT64, INT64], [0, 0], True, False, keys, limit,
                      out.data_ptr(), vout.data_ptr(), cap, stream.cuda_stream)
    return n


@pytest.mark.parametrize("groups", [1000, 62_500, 200_001])
def test_threads_and_streams(groups):
    dev = torch.device("cuda", 0)
    jobs = []
    for t in range(4):
        rng = np.random.default_rng(groups + t)
        words = np.zeros((groups, 2), np.int64)
        words[:, 0] = np.arange(groups) + 1
        words[:, 1] = rng.integers(-50, 50, groups)
        words[rng.random(groups) < 0.3] = 0  # absent groups
        present = words[words.any(axis=1)]
        order = np.lexsort((present[:, 0], present[:, 1] if t % 2 else -present[:, 1]))
        jobs.append((torch.from_numpy(words).to(dev), [(1, t % 2 == 0)], present[order]))
    torch.cuda.synchronize()
    failed = []

    def work(t):
        try:
            torch.cuda.set_device(0)
            src, keys, want = jobs[t]
            stream = torch.cuda.Stream()
            out = torch.empty(2 * groups, dtype=torch.int64, device=dev)
            vout = torch.empty(2 * ((groups + 63) // 64), dtype=torch.int64, device=dev)
            torch.cuda.synchronize()
            for _ in range(20):
                n = finalize(src, groups, keys, None, out, vout, stream)
                cols = out.cpu().numpy().reshape(2, groups)[:, :n].T
                if n != len(want) or not np.array_equal(cols, want):
                    failed.append((t, n, len(want)))
                    return
        except Exception as e:  # noqa: BLE001
            failed.append((t, repr(e)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    assert not failed
