"""CPU: the hand-over of item descriptions in the head-dim-256 kernel for one-tile items, as a model.

One warp of attend_tc5_wide_short_kernel writes the description of item n into slot n % 4 once `slot_free` says
that the slot's item before has been read.  The roles of a CTA are restated here with their barriers (a wait
passes once the phase of its parity has completed, as on the device) and run in random orders and with each role
in turn held back for as long as another one can go on.  In every order each role must see the items 0, 1, 2, ...
and none may get stuck.  How many arrivals complete `slot_free`, and which roles arrive on it, are read from the source."""
import random
import re
from pathlib import Path

import pytest

SLOTS = 4
SOURCE = Path(__file__).resolve().parent.parent / "baselinebenchmark_b200" / "csrc" / "attend_tc5.cu"


class Barrier:
    def __init__(self, count):
        self.count = self.left = count
        self.phase = 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def passed(self, parity):
        return (self.phase & 1) != parity


def slot_free_protocol():
    """(arrivals that complete a phase, the V warp is one of those that arrive)."""
    text = SOURCE.read_text()
    text = text[text.index("attend_tc5_wide_short_kernel(const Params p"):]
    text = text[:text.index("tmem_dealloc")]
    count = re.search(r"mbar_init\(smem_u32\(&c\.slot_free\[i\]\), (\d+)\)", text)
    sites = re.findall(r"if \(([^()]*)\) mbar_arrive\(smem_u32\(&c\.slot_free\[slot\]\)\)", text)
    assert "j == 0 && lane == 0" in sites                     # the softmax warps of the item
    return int(count.group(1)), "warp == 3 && lane == 0" in sites


class Model:
    """Roles are generators: they yield what they wait for, (barrier, parity), or None to let others run."""

    def __init__(self, items, count, v_arrives):
        self.items, self.v_arrives = items, v_arrives          # items: (key tiles, new K and V), then the end
        self.slot = [None] * SLOTS
        self.tensor_core = []                                  # barriers to arrive on, in order
        one = lambda n=1: Barrier(n)
        self.item_full = [one() for _ in range(SLOTS)]
        self.slot_free = [one(count) for _ in range(SLOTS)]
        self.q_full = one(4 + 1)                               # the copying warps and the K warp (one half stands for both)
        self.q_free, self.k_full, self.k_free, self.v_full, self.v_free = (one() for _ in range(5))
        self.s_full = [[one(), one()] for _ in range(2)]
        self.p_full = [one(4), one(4)]
        self.pv_full = [one(), one()]
        self.o_free = one(4)
        self.roles = {"describe": self.describe(), "mma": self.mma(), "k": self.k(), "v": self.v()}
        for w in range(8):
            self.roles[f"softmax{w}"] = self.softmax(w)

    def read(self, n):
        assert self.slot[n % SLOTS] == n, f"the description of item {self.slot[n % SLOTS]} in the place of item {n}"
        return self.items[n] if n < len(self.items) else None

    def described(self, n):
        return self.item_full[n % SLOTS], (n // SLOTS) & 1

    def describe(self):
        for n in range(len(self.items) + 2):                   # the end is published once for each warpgroup
            if n >= SLOTS:
                yield self.slot_free[n % SLOTS], (n // SLOTS - 1) & 1
            self.slot[n % SLOTS] = n
            yield None
            self.item_full[n % SLOTS].arrive()

    def k(self):
        kt = n = 0
        while True:
            yield self.described(n)
            item = self.read(n)
            if item is None:
                return
            if n > 0:
                yield self.q_free, (n - 1) & 1
            self.q_full.arrive()
            if item[1]:
                self.k_full.arrive()                           # (the copy lands at once)
            for _ in range(1, item[0]):
                yield self.k_free, kt & 1
                kt += 1
                self.k_full.arrive()
            n += 1

    def v(self):
        vt = n = 0
        while True:
            yield self.described(n)
            item = self.read(n)
            if item is None:
                return
            if self.v_arrives:
                self.slot_free[n % SLOTS].arrive()
            if item[1]:
                for _ in range(item[0]):
                    if vt > 0:
                        yield self.v_free, (vt - 1) & 1
                    vt += 1
                    self.v_full.arrive()
            n += 1

    def mma(self):
        tiles = []                                             # (item, tile, tiles, fresh) whose Q.K^T has been issued
        state = {"n": 0, "j": 0, "item": None, "kt": 0}

        def qk():
            n, j = state["n"], state["j"]
            if j == 0:
                yield self.described(n)
                state["item"] = self.read(n)
                if state["item"] is None:
                    return
                yield self.q_full, n & 1
            count, fresh = state["item"]
            if fresh:
                yield self.k_full, state["kt"] & 1
                state["kt"] += 1
            self.tensor_core += [self.s_full[n & 1][len(tiles) & 1], self.q_free if j + 1 == count else self.k_free]
            tiles.append((n, j, count, fresh))
            state["n"], state["j"] = (n + 1, 0) if j + 1 == count else (n, j + 1)

        yield from qk()
        at = vt = 0
        p_phase = [0, 0]
        while at < len(tiles):
            n, j, _, fresh = tiles[at]
            yield from qk()
            x = n & 1
            yield self.p_full[x], p_phase[x]
            p_phase[x] ^= 1
            if j == 0 and n > 0:
                yield self.o_free, (n - 1) & 1
            if fresh:
                yield self.v_full, vt & 1
                vt += 1
            if at + 1 < len(tiles) and tiles[at + 1][3]:
                self.tensor_core.append(self.v_free)
            self.tensor_core.append(self.pv_full[x])
            at += 1

    def softmax(self, w):
        x = w // 4

        def copy_rows(m):
            yield self.described(m)
            if self.read(m) is None:
                return
            yield None
            self.read(m)                                       # the offsets of its rows
            self.q_full.arrive()

        s_phase, pv_phase, tile0 = [0, 0], 0, 0
        if x == 1:
            yield from copy_rows(0)
        for n in range(x, len(self.items) + 2, 2):
            yield self.described(n)
            item = self.read(n)
            if item is None:
                return
            tile0 = sum(t for t, _ in self.items[:n])
            for j in range(item[0]):
                buf = (tile0 + j) & 1
                yield self.s_full[x][buf], s_phase[buf]
                s_phase[buf] ^= 1
                if j == 0:
                    self.slot_free[n % SLOTS].arrive()
                if j + 1 == item[0]:
                    yield from copy_rows(n + 1)
                if j > 0:
                    yield self.pv_full[x], pv_phase
                    pv_phase ^= 1
                self.p_full[x].arrive()
            yield self.pv_full[x], pv_phase
            pv_phase ^= 1
            self.o_free.arrive()

    def run(self, rng, held=None):
        waiting = {name: None for name in [*self.roles, "tensor core"]}
        while len(waiting) > 1:
            ready = [r for r, w in waiting.items()
                     if (self.tensor_core if r == "tensor core" else w is None or w[0].passed(w[1]))]
            assert ready, f"stuck: {sorted(waiting)}"
            ready = [r for r in ready if r != held] or ready
            name = rng.choice(ready)
            if name == "tensor core":
                self.tensor_core.pop(0).arrive()
                continue
            try:
                waiting[name] = next(self.roles[name])
            except StopIteration:
                del waiting[name]


ITEMS = {"one tile, runs on a chunk": [(1, n % 5 == 0) for n in range(30)],
         "one tile, one chunk for all": [(1, n == 0) for n in range(30)],
         "two tiles": [(2, True)] * 20,
         "mixed": [(1 + n % 2, True) for n in range(24)]}


@pytest.mark.parametrize("items", ITEMS.values(), ids=ITEMS)
def test_every_role_sees_the_items_in_order(items):
    count, v_arrives = slot_free_protocol()
    names = list(Model(items, count, v_arrives).roles) + ["tensor core", None]
    for seed in range(10):
        for held in names:
            Model(items, count, v_arrives).run(random.Random(seed), held)
