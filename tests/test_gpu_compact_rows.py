"""Compaction of so few and so many edited rows that a warp takes one, several
and thirty-two of them at a time."""
import numpy as np
import pytest

import streamgc_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exact,sorted_rows", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("n", [6, 31, 1000, 40001, 650003])
def test_every_edited_row_is_compacted(n, exact, sorted_rows):
    v = np.arange(n)
    g = S.Graph.from_edges(n, np.concatenate([np.stack([v, (v + d) % n], 1) for d in (1, 2)]))
    gone = v[: n - 1 : 2]  # each vertex (but for the odd ring's last) loses its edge to a neighbor
    ups = S.updates_from(np.stack([gone, gone + 1], 1), np.ones(len(gone)))
    mode = S.MODE_CONCURRENT if n > 1000 else S.MODE_DETERMINISTIC
    with S.StreamGC(g, exact_select=exact, sorted_rows=sorted_rows, max_batch=len(ups)) as h:
        h.apply(ups, mode)
        h.drain_and_compact()
        rp, col, hw = h.row_ptr().astype(np.int64), h.col(), h.highwater()
        want = g.degree.astype(np.int64)
        np.subtract.at(want, gone, 1)
        np.subtract.at(want, gone + 1, 1)
        assert np.array_equal(hw, want)
        for d in range(int(want.max())):  # slot d of every row that long: ascending, as the base rows were
            rows = np.nonzero(want > d)[0]
            ids = col[rp[rows] + d]
            assert (ids < n).all()
            if d:
                assert (ids > col[rp[rows] + d - 1]).all()
        rows = np.nonzero(want < rp[1:] - rp[:-1])[0]
        assert (col[rp[rows] + want[rows]] == 0xFFFFFFFF).all()
        assert h.check_state()["bad_rows"] == 0
