"""The order of a one-kernel repair's steps across blocks (sgc_kernels.cu
GridSync / repair_fused), checked on a model: every interleaving of a few
blocks that arrive at barriers, collect the next worklist and let block 0 decide
between sweeps. No sweep may lose an entry of the list collected by the one
before, a block that leaves the short sweeps to the first few may not clear a
recolored bit that those have set since, and no block may wait for good."""

BLOCKS = 3
TAIL_BLOCKS, TAIL_LIST = 2, 2  # lists of at most two entries go to two blocks


class Model:
    """Blocks as programs of atomic steps. A sweep k visits `lists[k]` vertices,
    recolors one of them (where `commits` says so; its bit lies in the last
    block's share of the whole grid's mask) and then collects lists[k + 1]
    vertices, spread over the blocks that run it.
    `reset`: where the list's count is made zero, 'serial' (by block 0 between
    two sweeps) or 'sweep' (by block 0 after the sweep's first barrier).
    `handoff`: how blocks leave, 'part' (block 0's decision, a last arrival that
    the others await) or 'go' (each by what it reads, unannounced)."""

    def __init__(self, lists, reset="serial", handoff="part", commits=()):
        self.lists, self.reset, self.handoff = lists, reset, handoff
        self.commits = list(commits) + [False] * len(lists)
        self.found = set()

    def start(self):
        shared = dict(count=0, gen=0, wl=self.lists[0], lim=self.lists[0], more=True, bit=0)
        if self.reset == "serial":
            shared["wl"] = 0
        return shared, [dict(pc="top", due=0, serials=0, k=0, nb=BLOCKS) for _ in range(BLOCKS)]

    def step(self, i, b, s):
        """One step of block i; False when it has to wait."""
        pc, last = b["pc"], b["nb"] - 1
        if pc == "top":  # the last block of those that ran the sweep clears the bit the sweep set
            b["pc"] = "read"
            if i == last and b["k"] and self.commits[b["k"] - 1]:
                s["bit"] = 0
        elif pc == "read":
            lim = s["lim"] if self.reset == "serial" else s["wl"]
            b["pc"] = "arrive"
            if not s["more"]:
                b["pc"] = "left"
            elif b["nb"] > TAIL_BLOCKS and lim <= TAIL_LIST:
                if self.handoff == "part":
                    b["due"] += b["nb"] - TAIL_BLOCKS
                b["nb"] = TAIL_BLOCKS
                if i >= TAIL_BLOCKS:
                    b["pc"] = "part" if self.handoff == "part" else "left"
        elif pc == "part":
            s["count"] += 1
            b["pc"] = "left"
        elif pc == "arrive":  # the barrier after the sweep's first pass
            s["count"] += 1
            b["due"] += b["nb"]
            b["pc"] = "wait"
        elif pc == "wait":
            if s["count"] < b["due"]:
                return False
            b["pc"] = "reset" if self.reset == "sweep" and i == 0 else "commit"
        elif pc == "reset":
            s["wl"] = 0
            b["pc"] = "commit"
        elif pc == "commit":
            b["pc"] = "collect"
            if self.commits[b["k"]]:
                if i == 0:
                    s["bit"] = 1
                b["pc"] = "arrive2"
        elif pc == "arrive2":
            s["count"] += 1
            b["due"] += b["nb"]
            b["pc"] = "wait2"
        elif pc == "wait2":
            if s["count"] < b["due"]:
                return False
            if i == last and not s["bit"]:
                self.found.add("lost bit")
            b["pc"] = "collect"
        elif pc == "collect":
            s["wl"] += sum(1 for e in range(self.lists[b["k"] + 1]) if e % b["nb"] == (i + 1) % b["nb"])
            b["pc"] = "arrive_serial"
        elif pc == "arrive_serial":
            s["count"] += 1
            b["due"] += b["nb"]
            b["serials"] += 1
            b["k"] += 1
            b["pc"] = "wait_all" if i == 0 else "wait_gen"
        elif pc == "wait_gen":
            if s["gen"] < b["serials"]:
                return False
            b["pc"] = "top"
        elif pc == "wait_all":
            if s["count"] < b["due"]:
                return False
            if s["wl"] != self.lists[b["k"]]:
                self.found.add("lost entry")
            s["more"] = b["k"] + 1 < len(self.lists)
            if self.reset == "serial":
                s["lim"], s["wl"] = s["wl"], 0
            s["gen"] += 1
            b["pc"] = "top"
        return True

    def explore(self):
        """Every order of the blocks' steps; what went wrong in any of them."""
        shared, blocks = self.start()
        todo, seen = [(shared, blocks)], set()
        while todo:
            shared, blocks = todo.pop()
            key = (tuple(shared.items()), tuple(tuple(b.items()) for b in blocks))
            if key in seen:
                continue
            seen.add(key)
            moved = False
            for i, b in enumerate(blocks):
                if b["pc"] == "left":
                    continue
                s2, b2 = dict(shared), dict(b)
                if self.step(i, b2, s2):
                    moved = True
                    todo.append((s2, blocks[:i] + [b2] + blocks[i + 1:]))
            if not moved and any(b["pc"] != "left" for b in blocks):
                self.found.add("stuck")
        return self.found


def test_no_entry_of_the_next_list_is_lost():
    for lists in ([5, 3, 0], [1, 1, 1, 0], [4, 0], [2, 6, 2, 0]):
        assert Model(lists).explore() == set()


def test_leaving_blocks_harm_nothing():
    for commits in ((True, True), (True, False, True), (False, True, True)):
        for lists in ([5, 2, 1, 0], [5, 4, 2, 0], [1, 4, 1, 0]):
            assert Model(lists, commits=commits).explore() == set()


def test_the_model_sees_a_reset_that_meets_an_add():
    assert Model([5, 3, 0], reset="sweep").explore() == {"lost entry"}


def test_the_model_sees_blocks_that_leave_unannounced():
    assert "lost bit" in Model([5, 2, 0], handoff="go", commits=(True, True)).explore()
    late = Model([5, 2, 4, 4, 0], handoff="go").explore()  # a late block reads the grown list and stays
    assert late == {"lost entry", "stuck"}
