"""Rows merged into one sorted run by a compaction, at row lengths on both sides
of the powers of two they are sorted at and of the longest row that is sorted."""
import numpy as np
import pytest

import streamgc_b200 as S

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 3, 31, 32, 33, 64, 65, 511, 513, 1023, 1024, 1025, 1500]


def test_rows_of_every_length_merge():
    hubs = len(LENGTHS)
    n = hubs + 2000
    rng = np.random.default_rng(1)
    start, later = [], []
    for k, length in enumerate(LENGTHS):  # a third of the row at creation, the rest inserted in random order
        ids = rng.permutation(np.arange(hubs, n))[:length]
        cut = (length + 2) // 3
        start.append(np.stack([np.full(cut, k), ids[:cut]], 1))
        later.append(np.stack([np.full(length - cut, k), ids[cut:]], 1))
    g = S.Graph.from_edges(n, np.concatenate(start))
    later = rng.permutation(np.concatenate(later))
    with S.StreamGC(g, exact_select=True, sorted_rows=True, max_batch=1 << 14) as h:
        h.apply(S.updates_from(later), S.MODE_CONCURRENT)
        h.repair()  # compacts every edited row
        rp, col, runs, hw = h.row_ptr(), h.col(), h.base_runs(), h.highwater()
        for k, length in enumerate(LENGTHS):
            row = col[int(rp[k]):int(rp[k]) + int(hw[k])]
            want = np.sort(np.concatenate([start[k][:, 1], later[later[:, 0] == k][:, 1]]))
            assert len(row) == length and np.array_equal(np.sort(row), want), length
            if length <= 1024:
                assert runs[k] == length and np.array_equal(row, want), length
        assert h.check_state()["bad_rows"] == 0
