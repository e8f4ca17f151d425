"""A host model of the dataflow Jacobi kernel's blocks (k_jacobi_flow in
fluid_gb300/csrc/k_pressure.cu): in each a thirteenth warp claims items, sends
for an item's w and w*b boxes once the sweeping warps have the item before it
in registers, for its phi box once the up to nine neighbours have published the
phase before, and publishes each tile after the warps have stored it -- the
next claim before that publication with two tiles or more a block, after it
with fewer.  One buffer, three barriers (full, empty, stored).  Random
interleavings of all blocks' actions check that every box is read while it
holds the right phase, that no store overwrites what a copy in flight still
reads, that the buffer is never filled while it is being read, and that
nothing deadlocks; and, with a tile that is never published, that every block
leaves with no phase of `full` left incomplete."""
import random

import pytest


def around(t, ntx, nty):
    ty, tx = divmod(t, ntx)
    return [y * ntx + x for y in range(max(0, ty - 1), min(nty, ty + 2))
            for x in range(max(0, tx - 1), min(ntx, tx + 2))]


class Flow:
    def __init__(self, ntx, nty, blocks, nphase, seed, stall=-1, ends_phase=True):
        self.rng = random.Random(seed)
        self.ntx, self.nty, self.stall, self.ends_phase = ntx, nty, stall, ends_phase
        self.nt = ntx * nty
        self.total, self.nphase = self.nt * nphase, nphase
        self.blocks = min(blocks, self.nt)
        self.done = [0] * self.nt
        self.buf = [[-1] * self.nt, [-1] * self.nt]
        self.reading = [[0] * self.nt, [0] * self.nt]
        self.counter = 0
        self.late = False  # the time limit of every wait has passed
        self.incomplete = 0

    def claim(self):
        self.counter += 1
        return self.counter - 1

    def ready(self, i):
        ph, t = divmod(i, self.nt)
        return all(self.done[n] >= ph for n in around(t, self.ntx, self.nty))

    def block(self):
        """[thirteenth warp, sweeping warps, the copies in flight]"""
        st = dict(full=0, empty=0, stored=0, arrivals=0, tx=0, item=0, lost=None, busy=False)
        flying = []

        def maybe_complete():
            if st["arrivals"] == 1 and st["tx"] == 0:
                st["full"] += 1
                st["arrivals"] = 0

        def send(i, box):
            ph, t = divmod(i, self.nt)
            assert not st["busy"], "a box lands in a buffer that is being read"
            if box == "phi":
                for n in around(t, self.ntx, self.nty):
                    assert self.buf[ph & 1][n] == ph - 1, "stale neighbour"
                    self.reading[ph & 1][n] += 1
            st["tx"] += 1
            flying.append((i, box))

        def copies():
            while True:
                if not flying:
                    yield False
                    continue
                i, box = flying.pop(self.rng.randrange(len(flying)))
                ph, t = divmod(i, self.nt)
                if box == "phi":
                    for n in around(t, self.ntx, self.nty):
                        self.reading[ph & 1][n] -= 1
                st["tx"] -= 1
                maybe_complete()
                yield True

        def arrive():
            st["arrivals"] += 1
            maybe_complete()

        def producer():
            deep = self.nt >= 2 * self.blocks
            nxt, cur, n = self.claim(), None, 0
            whole, flight = True, None
            while True:
                have = nxt < self.total
                taken, copied, told, ready = False, not have, cur is None, not have
                after = None
                while not (taken and copied and told):
                    moved = False
                    if not taken and (n == 0 or st["empty"] >= n):
                        taken = moved = True
                        st["item"] = nxt
                        if have:
                            flight, whole = n, False
                            send(nxt, "w")
                            send(nxt, "bw")
                        else:
                            arrive()
                    ready = ready or self.ready(nxt)
                    if not copied and ready and taken:
                        copied = whole = moved = True
                        if nxt >= self.nt:
                            send(nxt, "phi")
                        arrive()
                    if taken and not told and st["stored"] >= n:
                        if deep:
                            after = self.claim()
                        yield True
                        ph, t = divmod(cur, self.nt)
                        if t != self.stall:
                            self.done[t] = ph + 1
                        told = moved = True
                    if not moved and self.late:
                        if flight is not None:
                            if not whole and self.ends_phase:
                                st["lost"] = flight
                                arrive()
                            while st["full"] <= flight and (flying or st["arrivals"]):
                                yield True
                            self.incomplete += st["full"] <= flight
                        return
                    yield moved
                if not have:
                    return
                cur, n = nxt, n + 1
                nxt = self.claim() if n == 1 or not deep else after

        def warps():
            n = 0
            while True:
                while st["full"] <= n:
                    if self.late:
                        st["lost"] = n
                        return
                    yield False
                item = st["item"]
                if item >= self.total:
                    return
                st["busy"] = True
                yield True
                st["busy"] = False
                st["empty"] = n + 1
                yield True
                if st["lost"] is not None and st["lost"] <= n:
                    return
                ph, t = divmod(item, self.nt)
                assert not self.reading[1 - (ph & 1)][t], "overwrite before read"
                self.buf[1 - (ph & 1)][t] = ph
                yield True
                st["stored"] = n + 1
                n += 1

        return [producer(), warps()], copies()

    def run(self):
        actors = []
        live = 0
        for _ in range(self.blocks):
            a, c = self.block()
            actors += [[x, True] for x in a] + [[c, False]]
            live += len(a)
        idle = 0
        while live:
            k = self.rng.randrange(len(actors))
            it, counts = actors[k]
            try:
                moved = next(it)
            except StopIteration:
                actors[k] = actors[-1]
                actors.pop()
                live -= counts
                moved = True
            idle = 0 if moved else idle + 1
            if idle > 60 * len(actors):
                assert self.stall >= 0 and not self.late, "deadlock"
                self.late, idle = True, 0
        if self.stall < 0:
            assert self.done == [self.nphase] * self.nt
        return self.incomplete


SHAPES = [(19, 26, 152), (14, 19, 152), (1, 9, 4), (5, 5, 7), (3, 4, 12), (25, 7, 87)]


@pytest.mark.parametrize("ntx,nty,blocks", SHAPES)
def test_schedule_under_random_interleavings(ntx, nty, blocks):
    for seed in range(3):
        assert Flow(ntx, nty, blocks, 4, seed).run() == 0


@pytest.mark.parametrize("ntx,nty,blocks", SHAPES)
def test_blocks_leave_when_a_tile_is_never_published(ntx, nty, blocks):
    for seed in range(3):
        assert Flow(ntx, nty, blocks, 3, seed, stall=ntx * nty // 2).run() == 0


def test_the_model_sees_phases_left_incomplete():
    assert sum(Flow(5, 5, 7, 3, s, stall=12, ends_phase=False).run() for s in range(5)) > 0
