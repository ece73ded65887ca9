"""Passes over all rows where the hubs have neighboring ids, as graphs numbered by
degree have them: no slower than where the same hubs lie apart."""
import time

import numpy as np
import pytest

import streamgc_b200 as S

pytestmark = pytest.mark.gpu

N, HUBS, DEGREE = 200000, 64, 40000


@pytest.fixture(scope="module")
def graphs():
    """The same graph with hubs 0..63 and with hubs spread over the ids."""
    rng = np.random.default_rng(5)
    far = np.concatenate([rng.choice(np.arange(HUBS, N), DEGREE, replace=False) for _ in range(HUBS)])
    near = np.stack([np.repeat(np.arange(HUBS), DEGREE), far], 1)
    new_id = rng.permutation(N)
    return [(S.Graph.from_edges(N, e), e) for e in (near, new_id[near])]


def times(graphs, step):
    """Shortest of a few calls per graph."""
    out = []
    for g, edges in graphs:
        with S.StreamGC(g, exact_select=True, max_batch=1 << 18) as h:
            best = 1e9
            for _ in range(4):
                run = step(h, edges)
                h.synchronize()
                start = time.perf_counter()
                run()
                h.synchronize()
                best = min(best, time.perf_counter() - start)
            assert h.check_state()["bad_rows"] == 0
            out.append(best)
    return out


def test_forced_compaction(graphs):
    def step(h, edges):  # a change in every hub row and, through the other ends, in most others
        pick = edges[::7]
        for kind in (1, 0):
            ups = S.updates_from(pick, np.full(len(pick), kind))
            for k in range(0, len(ups), 1 << 18):
                h.apply(ups[k:k + (1 << 18)], S.MODE_CONCURRENT)
        return h.drain_and_compact
    near, apart = times(graphs, step)
    assert near < 2 * apart, (near, apart)


def test_validator(graphs):
    near, apart = times(graphs, lambda h, edges: h.validate)
    assert near < 2 * apart, (near, apart)
