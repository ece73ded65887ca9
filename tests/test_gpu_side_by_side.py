"""Handles side by side on one GPU: a publish does not wait for another handle's
long batch in stream order, and repairs of several handles in several threads
leave what each leaves alone."""
import threading
import time

import numpy as np
import pytest

import streamgc_b200 as S

pytestmark = pytest.mark.gpu


def hubs(n, seed):
    """A graph with a few long rows, so that updates of both ends take their time."""
    rng = np.random.default_rng(seed)
    e = np.stack([rng.integers(0, n, 8 * n), (rng.random(8 * n) ** 3 * n).astype(np.int64)], 1)
    return S.Graph.from_edges(n, e[e[:, 0] != e[:, 1]])


def test_publish_beside_a_long_batch_in_stream_order():
    ga, gb = hubs(16384, 1), hubs(24001, 2)
    ups = ga.churn_stream(32768, 50, 3)
    mine = gb.churn_stream(20 * 512, 50, 4)
    with S.StreamGC(ga, max_batch=len(ups)) as a, S.StreamGC(gb, exact_select=True) as b:
        b.publish()
        for k in range(4):  # first launches of everything
            b.apply(mine[k * 512:(k + 1) * 512], S.MODE_CONCURRENT)
            b.publish()
        a.apply(ups[:64], S.MODE_DETERMINISTIC)
        a.synchronize()
        start = time.perf_counter()
        a.apply(ups, S.MODE_DETERMINISTIC)  # returns before the GPU is done
        for k in range(4, 12):
            b.apply(mine[k * 512:(k + 1) * 512], S.MODE_CONCURRENT)
            assert b.publish()["proper"] == 1
        published = time.perf_counter() - start
        a.synchronize()
        assert published < 0.5 * (time.perf_counter() - start)


def test_repairs_of_several_handles_at_once():
    graphs = [hubs(n, n) for n in (300, 5000, 60000, 150001)]
    alone = []
    for g in graphs:
        with S.StreamGC(g, exact_select=True, full_repair_every=1) as h:
            h.publish()
            alone.append((h.colors(), h.bitmaps()))
    handles = [S.StreamGC(g, exact_select=True, full_repair_every=1) for g in graphs]
    wrong = []

    def work(h, want):
        for _ in range(6):
            h.upload("states", np.zeros(len(want[0]), np.uint32))
            if h.publish()["proper"] != 1 or not (np.array_equal(h.colors(), want[0]) and
                                                  np.array_equal(h.bitmaps(), want[1])):
                wrong.append(len(want[0]))

    threads = [threading.Thread(target=work, args=a) for a in zip(handles, alone)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for h in handles:
        assert h.stats()["device_error"] == 0
        h.close()
    assert not wrong
