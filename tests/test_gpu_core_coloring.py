"""The core coloring around its window of 128 vertices, against the greedy loop
it restates."""
import numpy as np
import pytest

import streamgc_b200 as S

pytestmark = pytest.mark.gpu


def greedy(g, colors, order):
    for v in order:
        if colors[v]:
            continue
        row = g.col_idx[int(g.row_ptr[v]):int(g.row_ptr[v + 1])]
        held = set(int(c) for c in colors[row])
        colors[v] = next((c for c in range(1, 2048) if c not in held), 2048)
    return colors


@pytest.mark.parametrize("n,dense", [(2, 1.0), (127, 0.5), (128, 1.0), (129, 0.9), (257, 0.3), (700, 0.05), (2100, 1.0)])
def test_core_coloring_is_the_greedy_loop(n, dense):
    rng = np.random.default_rng(n)
    a, b = np.triu_indices(n, 1)
    keep = rng.random(len(a)) < dense
    g = S.Graph.from_edges(n, np.stack([a[keep], b[keep]], 1))
    low = max(1, int(np.median(g.degree)))
    order = sorted((v for v in range(n) if g.degree[v] >= low), key=lambda v: (-int(g.degree[v]), v))
    with S.StreamGC(g, exact_select=True) as h:
        given = np.where(rng.random(n) < 0.1, rng.integers(1, 40, n), 0).astype(np.uint32)  # some colored before
        h.upload("states", given)
        want = greedy(g, given.astype(np.int64), order)
        assert h.color_core(low) == sum(1 for v in order if not given[v])
        assert np.array_equal(h.colors(), want)
        assert h.color_core(low) == 0 and np.array_equal(h.colors(), want)
