"""The repair as one kernel against the same passes as kernels of their own
(which timed handles run), array by array, around the sizes where it goes from
the whole grid to a few blocks and where it leaves a sweep to the others."""
import numpy as np
import pytest

import streamgc_b200 as S

pytestmark = pytest.mark.gpu


def graph(n, seed):
    """A ring with random chords and, where there is room, hub rows on both sides
    of the per-thread limit (64 slots) and of one and two work items (512)."""
    rng = np.random.default_rng(seed)
    v = np.arange(n)
    e = [np.stack([v, (v + 1) % n], 1), rng.integers(0, n, (n, 2))]
    for k, deg in enumerate((64, 65, 511, 513, 5000)):
        if deg < n // 2:
            e.append(np.stack([np.full(deg, k), rng.choice(np.arange(8, n), deg, replace=False)], 1))
    e = np.concatenate(e)
    return S.Graph.from_edges(n, e[e[:, 0] != e[:, 1]])


@pytest.mark.parametrize("exact", [True, False], ids=["exact", "reference"])
@pytest.mark.parametrize("n", [3, 33, 2047, 2049, 40000, (1 << 19) - 1, (1 << 19) + 1])
def test_same_as_the_separate_kernels(n, exact):
    g = graph(n, n)
    churn = g.churn_stream(min(2 * n, 20000), 50, 3)
    with S.StreamGC(g, exact_select=exact, profile=True, full_repair_every=2) as a, \
            S.StreamGC(g, exact_select=exact, full_repair_every=2) as b:
        for k in range(4):  # from no color, then after updates: full and incremental repairs
            ra, rb = a.publish(), b.publish()
            assert ra == rb
            for what in ("states", "bitmaps", "snapshot", "col"):
                assert np.array_equal(getattr(a, what)(), getattr(b, what)()), (k, what)
            sa, sb = a.stats(), b.stats()
            assert sa["live_entries"] == sb["live_entries"] and sb["device_error"] == 0
            part = churn[k * 4096:(k + 1) * 4096]
            a.apply(part, S.MODE_DETERMINISTIC)
            b.apply(part, S.MODE_DETERMINISTIC)


@pytest.mark.parametrize("exact", [True, False], ids=["exact", "reference"])
@pytest.mark.parametrize("n", [33, 2049, 40000, 250007, (1 << 19) - 1, (1 << 19) + 1])
def test_same_from_conflicting_colors(n, exact):
    """Colors drawn at random: many conflicts, sweeps that recolor in every size
    of list from all vertices down to a few."""
    g = graph(n, n)
    with S.StreamGC(g, exact_select=exact, profile=True) as a, S.StreamGC(g, exact_select=exact) as b:
        for top in (2, 12, 200):
            states = np.random.default_rng(top).integers(0, top + 1, n).astype(np.uint32)
            for h in (a, b):
                h.upload("states", states)
            ra, rb = a.publish(), b.publish()
            assert ra == rb and rb["proper"] == 1
            for what in ("states", "bitmaps", "snapshot"):
                assert np.array_equal(getattr(a, what)(), getattr(b, what)()), (top, what)
            assert b.stats()["device_error"] == 0


@pytest.mark.parametrize("cuda_graph", [True, False])
def test_batch_of_more_vertices_than_one_kernel_sweeps(cuda_graph):
    """The first tick's sweeps visit more than 2^19 vertices: the loop goes on in
    the captured while-node (or from the host). Each graph's colors are those it
    gets alone."""
    graphs = [graph(n, n) for n in (250007, 300001, 40000)]
    alone = []
    for g in graphs:
        with S.StreamGC(g, exact_select=True) as h:
            assert h.publish()["proper"] == 1
            alone.append(h.snapshot())
    b = S.Batch(graphs, epoch_sizes=[1024] * 3, cuda_graph=cuda_graph)
    try:
        b.close_epochs()
        assert b.tick()["proper"] == 1
        for k, want in enumerate(alone):
            assert np.array_equal(b.snapshot(k), want), k
    finally:
        b.close()


# the marks read sixteen bytes per lane by the first blocks (over 786,432 vertices)
# and by the whole grid (over 7,077,888), the last size the first blocks take
# (3,145,728) and the next
@pytest.mark.parametrize("n", [786465, 3145728, 3145729, 7077921])
def test_same_with_masks_of_many_words(n):
    v = np.arange(n)
    g = S.Graph.from_edges(n, np.concatenate([np.stack([v, (v + d) % n], 1) for d in (1, 5)]))
    with S.StreamGC(g, exact_select=True, profile=True, full_repair_every=0) as a, \
            S.StreamGC(g, exact_select=True, full_repair_every=0) as b:
        states = np.random.default_rng(n).integers(0, 4, n).astype(np.uint32)
        for h in (a, b):
            h.upload("states", states)
        churn = g.churn_stream(3 * 3000, 50, 3)
        last = S.updates_from(np.array([[n - 2, n - 1], [n - 1, 0]]), np.ones(2))  # the last word too
        for k in range(4):
            ra, rb = a.publish(), b.publish()
            assert ra == rb and rb["incremental"] == (k > 0)
            for what in ("states", "bitmaps", "snapshot"):
                assert np.array_equal(getattr(a, what)(), getattr(b, what)()), (k, what)
            for h in (a, b):
                h.apply(np.concatenate([churn[k * 3000:(k + 1) * 3000], last]), S.MODE_DETERMINISTIC)
