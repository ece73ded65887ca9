"""Stream-order updates (the reference's rules and the batched form's) on graphs
so small that nearly every update meets a row edited moments before: the
applying warp then has to settle what the preparing warps found. Compared with
the oracle array by array."""
import numpy as np
import pytest

import streamgc_b200 as S
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def hot_updates(n, count, seed, out_of_range):
    """Random updates over few vertices: repeats of one edge, absent deletes,
    present inserts, self loops and (optionally) endpoints outside the graph."""
    rng = np.random.default_rng(seed)
    pairs = rng.integers(0, n + (2 if out_of_range else 0), (count, 2))
    pairs[::7] = pairs[0] % n  # one edge again and again
    pairs[3::11, 1] = pairs[3::11, 0]  # self loops
    types = (rng.random(count) < 0.45).astype(np.uint8)
    types[5::97] = 7  # neither kind
    return S.updates_from(pairs, types)


# n, degree, slack, threshold: rows that overflow, rows on both sides of 64 slots
# (loaded whole or searched) and of 256 (several rounds), histogram rows
SHAPES = [(2, 1, 0, 64), (7, 3, 0, 2), (40, 20, 100, 8), (96, 70, 30, 64), (400, 300, 50, 64)]


@pytest.mark.parametrize("count", [1, 8, 9, 10, 14, 15, 16, 19, 31, 4000])  # around the chunks of 9
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: f"n{s[0]}")
def test_hot_rows_match_the_oracle(shape, count):
    n, degree, slack, thr = shape
    rng = np.random.default_rng(n)
    g = S.Graph.from_edges(n, np.stack([rng.integers(0, n, n * degree // 2 + 1) for _ in range(2)], 1))
    ups = np.concatenate([g.init_stream(), hot_updates(n, count, count, True)])
    o = O.Oracle(g.row_ptr, g.col_idx, g.degree, hist_threshold=thr, slack_pct=slack)
    with S.StreamGC(g, histogram_threshold=thr, slack_pct=slack, max_batch=len(ups)) as h:
        for part in (ups, hot_updates(n, count, count + 1, False)):
            h.apply(part[: len(ups)], S.MODE_DETERMINISTIC)
            o.apply(part[: len(ups)])
            for name, a, b in (("states", h.states(), o.states()), ("bitmaps", h.bitmaps(), o.bitmaps()),
                               ("col", h.col(), o.col()), ("hist", h.hist(), o.hist())):
                assert np.array_equal(a, b), name
            assert h.check_state()["bad_rows"] == 0
            h.epoch()
            o.epoch()
            assert np.array_equal(h.col(), o.col()) and np.array_equal(h.bitmaps(), o.bitmaps())
