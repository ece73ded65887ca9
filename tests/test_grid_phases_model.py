"""The order of a one-kernel repair's steps across blocks (sgc_kernels.cu
GridSync / repair_fused), checked on a model: every interleaving of a few
blocks that arrive at barriers, collect the next worklist and let block 0 decide
between sweeps. No sweep may lose an entry of the list collected by the one
before."""

BLOCKS = 3


class Model:
    """Blocks as programs of atomic steps. A sweep k visits `lists[k]` vertices
    and then collects lists[k + 1] of them, spread over the blocks that run it.
    `reset`: where the list's count is made zero, 'serial' (by block 0 between
    two sweeps) or 'sweep' (by block 0 after the sweep's first barrier)."""

    def __init__(self, lists, reset):
        self.lists, self.reset = lists, reset
        self.found = set()

    def start(self):
        shared = dict(count=0, gen=0, wl=self.lists[0], lim=self.lists[0], more=True)
        if self.reset == "serial":
            shared["wl"] = 0
        return shared, [dict(pc="top", due=0, serials=0, k=0, nb=BLOCKS) for _ in range(BLOCKS)]

    def step(self, i, b, s):
        """One step of block i; False when it has to wait."""
        pc = b["pc"]
        if pc == "top":
            if not s["more"]:
                b["pc"] = "left"
                return True
            b["pc"] = "arrive"
        elif pc == "arrive":  # the barrier after the sweep's first pass
            s["count"] += 1
            b["due"] += b["nb"]
            b["pc"] = "wait"
        elif pc == "wait":
            if s["count"] < b["due"]:
                return False
            b["pc"] = "reset" if self.reset == "sweep" and i == 0 else "collect"
        elif pc == "reset":
            s["wl"] = 0
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
        assert Model(lists, "serial").explore() == set()


def test_the_model_sees_a_reset_that_meets_an_add():
    assert Model([5, 3, 0], "sweep").explore() == {"lost entry"}
