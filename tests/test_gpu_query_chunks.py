"""Point queries at and around the number of vertices one launch answers."""
import numpy as np
import pytest

import streamgc_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 255, 257, 65535, 65536, 65537, 140000])
def test_queries_of_every_size_read_the_snapshot(k):
    n = 5000
    v = np.arange(n)
    g = S.Graph.from_edges(n, np.stack([v, (v + 1) % n], 1))
    rng = np.random.default_rng(k)
    with S.StreamGC(g, exact_select=True) as h:
        h.publish()
        snap = h.snapshot()
        for _ in range(2):
            q = rng.integers(0, n + 50, k).astype(np.uint32)  # ids outside the graph answer 0
            want = np.where(q < n, snap[np.minimum(q, n - 1)], 0)
            assert np.array_equal(h.query(q), want)
