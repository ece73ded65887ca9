"""The validator on rows with repeated, one-sided and self entries, against sets
of edges."""
import numpy as np
import pytest

import streamgc_b200 as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 33, 256, 257, 4096])
def test_validator_counts_distinct_edges(n):
    rng = np.random.default_rng(n)
    rows = [rng.integers(0, n, rng.integers(0, 40)) for _ in range(n)]  # repeats, self entries, one-sided
    rows[-1] = np.append(rows[-1], [n - 1, n - 1, 0])
    rp = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    g = S.Graph(rp, np.concatenate(rows))
    colors = rng.integers(0, 6, n)
    edges = {(min(x, int(y)), max(x, int(y))) for x, r in enumerate(rows) for y in r}
    with S.StreamGC(g) as h:
        h.upload("states", colors.astype(np.uint32))
        for _ in range(2):
            v = h.validate()
            assert v["edges"] == len(edges)
            assert v["violations"] == sum(1 for a, b in edges if colors[a] == colors[b] != 0)
            assert v["uncolored_with_edges"] == sum(1 for x, r in enumerate(rows) if len(r) and not colors[x])
            assert v["max_color"] == colors.max() and v["out_of_range"] == 0
