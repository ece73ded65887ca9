"""The work a program has this framework do, as cases that can be timed.

Each case is a dict of plain values. `prepare` builds what a program holds
before the call (a graph resident in a handle, colored, and the updates that
will arrive), `run` makes one pass through the public entry points and returns
the colors that pass leaves, `work` counts the bytes the pass cannot do without.

Graphs come from the three families of the benchmark: a planar triangulation
(`mesh`: even degrees of about 6), R-MAT with (a, b, c) = (.57, .19, .19)
(`rmat`: dense hubs) and Chung-Lu with exponent 2.1 and degrees capped at
100,000 (`power`: long hub rows, ids in order of expected degree). They are
drawn on the GPU.

Updates form a ring: every chosen edge is deleted once and inserted once per
turn, at random places, half the updates being inserts. Every update changes
the graph, and after a turn the rows hold the same edges again, so a state can
be run as often as wanted. All outputs are whole numbers.
"""
import math

import numpy as np
import torch

import streamgc_b200 as S

DEVICE = "cuda:0"
CORE_DEGREE = 256  # vertices colored one at a time before the first repair of a loaded graph


def listed():
    return [
        # A reader asks for the colors of a few vertices of the published snapshot.
        dict(name="query", kind="query", family="mesh", n=131072, degree=6, points=257),
        # The reference's protocol, the default of every stepping call: one short batch
        # in stream order, then the epoch's maintenance, on a graph with hubs.
        dict(name="det_epoch", kind="det", family="rmat", n=16384, degree=16, epoch=8192, ring=4),
        # The concurrent mode of a handle made with the default options (the
        # reference's rules: histograms above the threshold, every vertex swept).
        dict(name="conc_default", kind="conc", family="mesh", n=65536, degree=6, epoch=8192, ring=8, epochs=8,
             exact=False, captured=False, sorted_rows=False, feed="host", full_every=16),
        # The benchmark's small workload: a Delaunay-like graph, updates from pinned
        # host memory, the captured publish.
        dict(name="conc_mesh", kind="conc", family="mesh", n=131072, degree=6, epoch=32768, ring=8, epochs=8,
             exact=True, captured=True, sorted_rows=False, feed="pinned", full_every=0),
        # Short epochs, where each one is mostly launches: the shortest of the
        # benchmark's epoch sizes, eager publishes, ordinary host arrays.
        dict(name="conc_mesh_short", kind="conc", family="mesh", n=24001, degree=6, epoch=4096, ring=8, epochs=8,
             exact=True, captured=False, sorted_rows=False, feed="host", full_every=16),
        # Rows kept sorted, the default cadence of full repairs, hubs, ragged sizes.
        dict(name="conc_power_sorted", kind="conc", family="power", n=300007, degree=17, epoch=50021, ring=8, epochs=8,
             exact=True, captured=False, sorted_rows=True, feed="host", full_every=16),
        # The benchmark's skewed workload: R-MAT with a dense core, updates inside
        # the core, already on the GPU.
        dict(name="conc_rmat_core", kind="conc", family="rmat", n=1 << 20, degree=64, epoch=65536, ring=16, epochs=16,
             exact=True, captured=True, sorted_rows=False, feed="device", full_every=0, core=True),
        # The benchmark's large workload at a size that is quick to build: a power-law
        # graph with rows up to 100,000 entries, the longest epoch of its sweep.
        dict(name="conc_power_large", kind="conc", family="power", n=2000003, degree=55, epoch=262144, ring=8, epochs=4,
             exact=True, captured=True, sorted_rows=False, feed="pinned", full_every=0),
        # The end of a phase: the last batches, a full repair, the validator, the
        # coloring downloaded for the output files.
        dict(name="phase_end", kind="phase", family="rmat", n=1 << 18, degree=32, epoch=65536, ring=8, epochs=4),
        # Loading a graph without its init stream: the core's coloring, then the first
        # publish repairs every vertex.
        dict(name="load_color", kind="load", family="power", n=300007, degree=17),
        # The batched engine: one epoch of each of many uneven graphs per tick.
        dict(name="batch_tick", kind="batch", graphs=24, n_lo=1024, n_hi=262144, ring=8, epochs=4),
        # A server of small tenants whose results must not depend on the mix.
        dict(name="serve_tenants", kind="serve", graphs=32, n_lo=512, n_hi=8192, ring=8, epochs=4),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["query", "det", "conc", "conc", "conc", "conc", "phase", "load", "batch", "serve"])
    family = rng.choice(["mesh", "rmat", "power"])
    degree = 6 if family == "mesh" else rng.randint(8, 40)
    if kind == "query":
        return dict(kind=kind, family=family, n=size(4096, 400000), degree=degree, points=size(1, 65536))
    if kind == "det":
        n = size(2048, 24000)
        return dict(kind=kind, family=family, n=n, degree=min(degree, 16), epoch=size(256, min(8192, n // 2)), ring=4)
    if kind == "phase":
        n = size(50000, 300000)
        return dict(kind=kind, family=family, n=n, degree=min(degree, 32), epoch=size(n // 8, n // 4), ring=4, epochs=4)
    if kind == "load":
        return dict(kind=kind, family=family, n=size(8192, 300000), degree=min(degree, 24))
    if kind == "batch":
        return dict(kind=kind, graphs=rng.randint(5, 32), n_lo=size(600, 1200), n_hi=size(30000, 200000), ring=4,
                    epochs=rng.randint(1, 4))
    if kind == "serve":
        return dict(kind=kind, graphs=rng.randint(8, 60), n_lo=size(500, 700), n_hi=size(3000, 9000), ring=4,
                    epochs=rng.randint(1, 4))
    if rng.random() < 0.15:
        n = size(8192, 60000)
        return dict(kind=kind, family="mesh", n=n, degree=6, epoch=size(n // 32, n // 8), ring=8, epochs=8,
                    exact=False, captured=False, sorted_rows=False, feed="host", full_every=16)
    n = size(16384 if family == "mesh" else 65536, 1000000)
    return dict(kind=kind, family=family, n=n, degree=degree, epoch=min(131072, size(n // 8, n // 4)), ring=4,
                epochs=8, exact=True, captured=rng.random() < 0.6, sorted_rows=rng.random() < 0.3,
                feed=rng.choice(["host", "pinned", "device"]), full_every=rng.choice([0, 16]))


# ---- inputs ----

def _edges(family, n, degree, gen):
    """Distinct undirected edges of a graph of the family, as keys a * n + b with a < b, ascending."""
    if family == "mesh":  # a grid with one random diagonal per cell, ids shuffled
        w = max(2, math.isqrt(n - 1) + 1)
        v = torch.arange(n, device=DEVICE)
        inside = v % w != w - 1
        right, down = v[inside], v
        diag = v[inside]
        flip = torch.rand(len(diag), generator=gen, device=DEVICE) < 0.5
        da = torch.where(flip, diag, diag + 1)
        db = torch.where(flip, diag + w + 1, diag + w)
        a, b = torch.cat([right, down, da]), torch.cat([right + 1, down + w, db])
        keep = b < n
        perm = torch.randperm(n, generator=gen, device=DEVICE)
        a, b = perm[a[keep]], perm[b[keep]]
    elif family == "rmat":  # degree / 2 draws per vertex
        m, levels = n * degree // 2, max(1, math.ceil(math.log2(n)))
        a = torch.zeros(m, dtype=torch.int64, device=DEVICE)
        b = torch.zeros(m, dtype=torch.int64, device=DEVICE)
        for _ in range(levels):
            r = torch.rand(m, generator=gen, device=DEVICE)
            a = 2 * a + (r >= 0.76)
            b = 2 * b + (((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        keep = (a < n) & (b < n)
        a, b = a[keep], b[keep]
    else:  # power: endpoints drawn with probability proportional to the expected degrees
        w = torch.arange(1, n + 1, dtype=torch.float64, device=DEVICE) ** (-1.0 / 1.1)
        scale = degree * n / float(w.sum())
        for _ in range(30):
            scale *= degree * n / float((w * scale).clamp(max=100000.0).sum())
        cum = (w * scale).clamp(max=100000.0).cumsum(0)
        m = n * degree // 2
        ends = torch.rand(2 * m, generator=gen, dtype=torch.float64, device=DEVICE) * cum[-1]
        ends = torch.searchsorted(cum, ends).clamp(max=n - 1)
        a, b = ends[:m], ends[m:]
    keep = a != b
    a, b = a[keep], b[keep]
    return torch.unique(torch.minimum(a, b) * n + torch.maximum(a, b))


def _graph(keys, n):
    """The host CSR of edges a * n + b, rows ascending."""
    a, b = keys // n, keys % n
    both = torch.cat([keys, b * n + a]).sort().values
    rows = torch.zeros(n + 1, dtype=torch.int64, device=DEVICE)
    rows[1:] = torch.bincount(both // n, minlength=n).cumsum(0)
    return S.Graph(rows.cpu().numpy(), (both % n).to(torch.int32).cpu().numpy().view(np.uint32))


def _ring(family, n, degree, length, gen, core=False):
    """A graph and `length` updates (even) that lead back to it: each chosen edge
    has one DEL and one ADD at random places; edges whose ADD comes first are
    absent at the start. With `core`, the chosen edges join vertices of the top
    tenth by degree. Each edge is listed in a random direction per update."""
    keys = _edges(family, n, degree, gen)
    pool = torch.arange(len(keys), device=DEVICE)
    if core:
        deg = torch.bincount(torch.cat([keys // n, keys % n]), minlength=n)
        floor = deg.sort().values[(9 * n) // 10]
        pool = pool[(deg[keys // n] >= floor) & (deg[keys % n] >= floor)]
    picks = min(length // 2, len(pool) // 2)
    chosen = pool[torch.randperm(len(pool), generator=gen, device=DEVICE)[:picks]]
    place = torch.randperm(2 * picks, generator=gen, device=DEVICE).view(2, picks)
    absent = torch.rand(picks, generator=gen, device=DEVICE) < 0.5
    first, second = place.min(0).values, place.max(0).values
    key = torch.empty(2 * picks, dtype=torch.int64, device=DEVICE)
    add = torch.empty(2 * picks, dtype=torch.bool, device=DEVICE)
    key[first], key[second] = keys[chosen], keys[chosen]
    add[first], add[second] = absent, ~absent
    turn = torch.rand(2 * picks, generator=gen, device=DEVICE) < 0.5
    a, b = key // n, key % n
    pairs = torch.stack([torch.where(turn, b, a), torch.where(turn, a, b)], 1)
    start = torch.ones(len(keys), dtype=torch.bool, device=DEVICE)
    start[chosen[absent]] = False
    updates = S.updates_from(pairs.cpu().numpy().astype(np.uint32), (~add).to(torch.uint8).cpu().numpy())
    return _graph(keys[start], n), updates


def _many(case, gen):
    """Uneven graphs, log-uniform in size, families in turn, with the updates of their epochs."""
    rng = np.random.default_rng(case["graphs"])
    graphs, rings, epochs = [], [], []
    for k in range(case["graphs"]):
        n = int(round(math.exp(rng.uniform(math.log(case["n_lo"]), math.log(case["n_hi"])))))
        family = ("mesh", "rmat", "power")[k % 3]
        epoch = max(64, min(8192, 1 << int(math.log2(n / 8)))) if case["kind"] == "batch" else int(rng.integers(16, 257))
        g, ups = _ring(family, n, 6 if family == "mesh" else 16, epoch * case["ring"], gen)
        graphs.append(g)
        rings.append(ups)
        epochs.append(min(epoch, len(ups)))
    return graphs, rings, epochs


def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind = case["kind"]
    state = dict(case=case, at=0)
    if kind in ("batch", "serve"):
        graphs, state["rings"], state["epochs"] = _many(case, gen)
        state["turn"] = [0] * len(graphs)
        if kind == "batch":
            b = state["batch"] = S.Batch(graphs, epoch_sizes=state["epochs"], max_tick_updates=1 << 18)
            b.close_epochs()
            b.color_core(CORE_DEGREE)
            b.tick()
        else:
            srv = state["server"] = S.Server(hbm_budget_bytes=16 << 30, max_tick_updates=1 << 16, stream_order=True)
            state["tenants"] = [srv.add_tenant(g, epoch_size=e) for g, e in zip(graphs, state["epochs"])]
            srv.step()
        return state

    n, family, degree = case["n"], case["family"], case["degree"]
    if kind in ("query", "load"):
        graph, ups = _graph(_edges(family, n, degree, gen), n), None
    else:
        graph, ups = _ring(family, n, degree, case["epoch"] * case["ring"], gen, case.get("core", False))
        state["epoch"] = min(case["epoch"], len(ups))
        state["batches"] = [ups[i:i + state["epoch"]] for i in range(0, len(ups) - state["epoch"] + 1, state["epoch"])]
        if len(ups) % state["epoch"]:  # the rest of the turn: the ring has to close
            state["batches"].append(ups[len(state["batches"]) * state["epoch"]:])
    if kind == "det" or (kind == "conc" and not case["exact"]):  # colored through its init stream, as the reference does
        h = S.StreamGC(graph, epoch_size=state["epoch"])
        h.process_stream(graph.init_stream(), S.MODE_DETERMINISTIC)
        h.repair()
    else:
        h = S.StreamGC(graph, epoch_size=state.get("epoch", 32768), max_batch=state.get("epoch", 32768),
                       exact_select=True, graph_publish=case.get("captured", False),
                       sorted_rows=case.get("sorted_rows", False), full_repair_every=case.get("full_every", 16))
        h.color_core(CORE_DEGREE)
        h.publish()
    state["handle"] = h
    if kind == "query":
        state["points"] = np.random.default_rng([seed, 3]).integers(0, n, case["points"]).astype(np.uint32)
    elif kind == "load":
        state["uncolored"] = np.zeros(n, dtype=np.uint32)
    elif kind == "phase" or case.get("feed") in ("pinned", "device"):
        feed = torch.from_numpy(ups.view(np.uint8))
        state["feed"] = feed.to(DEVICE) if case.get("feed") == "device" else feed.pin_memory()
    for name, size in (("words", 4), ("bitmaps", 8)) if kind == "det" else (("colors", 2),):
        state[name] = torch.zeros(size * n, dtype=torch.uint8).pin_memory()
    return state


# ---- one pass ----

def _download(state, what, into, dtype):
    buf = state[into]
    state["handle"].download_into(what, buf.data_ptr(), buf.numel())
    return buf.numpy().view(dtype)


def _next(state):
    """The next batch of the ring: its index, and the address of its updates where they sit in pinned or device memory."""
    k = state["at"]
    state["at"] = (k + 1) % len(state["batches"])
    feed = state.get("feed")
    return state["batches"][k], (feed.data_ptr() + 16 * k * state["epoch"]) if feed is not None else 0


def run(state):
    kind, h = state["case"]["kind"], state.get("handle")
    if kind == "query":
        return h.query(state["points"])
    if kind == "det":
        batch, _ = _next(state)
        h.apply(batch, S.MODE_DETERMINISTIC)
        h.epoch()
        return _download(state, "states", "words", "<u4"), _download(state, "bitmaps", "bitmaps", "<u8").view("<i8")
    if kind == "conc":
        proper = 1
        for _ in range(state["case"]["epochs"]):
            batch, ptr = _next(state)
            if ptr:
                h.apply_ptr(ptr, len(batch), S.MODE_CONCURRENT)
            else:
                h.apply(batch, S.MODE_CONCURRENT)
            proper &= h.publish()["proper"]
        return _download(state, "snapshot", "colors", "<u2"), proper
    if kind == "phase":
        for _ in range(state["case"]["epochs"]):
            batch, ptr = _next(state)
            h.apply_ptr(ptr, len(batch), S.MODE_CONCURRENT)
        report = h.repair()
        check = h.validate()
        return (_download(state, "colors", "colors", "<u2"), report["proper"], check["violations"], check["edges"],
                check["uncolored_with_edges"])
    if kind == "load":
        h.upload("states", state["uncolored"])
        core = h.color_core(CORE_DEGREE)
        report = h.publish()
        return _download(state, "snapshot", "colors", "<u2"), core, report["proper"]
    for _ in range(state["case"]["epochs"]):
        for k, ups in enumerate(state["rings"]):
            t, e = state["turn"][k], state["epochs"][k]
            part = ups[t:t + e]
            state["turn"][k] = t + e if t + e < len(ups) else 0
            if kind == "batch":
                state["batch"].submit(k, part)
            else:
                state["server"].submit(state["tenants"][k], part)
        if kind == "batch":
            state["batch"].tick()
        else:
            state["server"].step()
    if kind == "batch":
        return np.concatenate([state["batch"].snapshot(k) for k in range(len(state["rings"]))])
    return np.concatenate([state["server"].snapshot(t) for t in state["tenants"]])


# ---- what a pass cannot do without ----

# Per update: its record (16 B) and, at both endpoints, the row's bounds and
# marks (24 B), the slot read and written (8 B), the state word (4 B) and the
# bitmap read and written (16 B).
UPDATE_BYTES = 16 + 2 * (24 + 8 + 4 + 16)
# A pass over every row: 8 B per entry (the entry and its neighbor's color), and
# per vertex the row's bounds, marks and class, the state word and the bitmap.
ENTRY_BYTES, VERTEX_BYTES = 8, 36


def work(case):
    kind = case["kind"]
    if kind == "query":
        return dict(bytes=8 * case["points"], flops=0)
    if kind in ("batch", "serve"):
        mean = (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])  # of a log-uniform size
        epoch = min(8192, mean / 12) if kind == "batch" else 136
        return dict(bytes=case["graphs"] * (case["epochs"] * epoch * UPDATE_BYTES + 2 * mean), flops=0)
    n = case["n"]
    sweep = n * (case["degree"] * ENTRY_BYTES + VERTEX_BYTES)
    if kind == "load":
        return dict(bytes=sweep + 6 * n, flops=0)
    updates = case["epoch"] * UPDATE_BYTES
    if kind == "phase":  # the repair's sweep and the validator's pass over the rows
        return dict(bytes=case["epochs"] * updates + 2 * sweep + 2 * n, flops=0)
    if kind == "det":  # every bitmap is rebuilt from the rows
        return dict(bytes=updates + sweep + 12 * n, flops=0)
    # every epoch's updates; under the default rules every row is swept too
    return dict(bytes=case["epochs"] * (updates + (0 if case["exact"] else sweep)) + 2 * n, flops=0)
