"""How a block of the dataflow Jacobi kernel (k_jacobi_flow in
fluid_gb300/csrc/k_pressure.cu) ends when waits give up: twelve sweeping warps
and the warp that claims items, copies and publishes, run action by action in
random order.  A wait may give up at any time from a random moment on.  The
twelve warps meet in barriers that all of them must reach; nothing may be left
waiting in one, and no warp may store an item that another has given up on."""
import random

import pytest

WARPS, SWEEPS = 12, 8


class Block:
    def __init__(self, items, rng, agree=True, named=True):
        """agree: a warp that has seen the end passes the barriers too; named:
        the mark of a warp that gave up says on which item."""
        self.items, self.rng, self.agree, self.named = items, rng, agree, named
        self.full = self.empty = self.stored = 0  # completed phases
        self.n_empty = self.n_stored = 0          # arrivals of the present phase
        self.item, self.lost = 0, None
        self.at_barrier, self.passed = 0, 0
        self.impatient = rng.random() < 0.7
        self.when = rng.randrange(1, 60 * WARPS * (items + 1))
        self.clock = 0
        self.stores = [0] * (items + 1)

    def gives_up(self):
        return self.impatient and self.clock >= self.when and self.rng.random() < 0.3

    def wait(self, done):
        while not done():
            if self.gives_up():
                return False
            yield
        return True

    def barrier(self):
        mine = self.passed
        self.at_barrier += 1
        if self.at_barrier == WARPS:
            self.at_barrier, self.passed = 0, self.passed + 1
        while self.passed == mine:
            yield "barrier"

    def producer(self):
        for n in range(self.items + 1):
            if n:
                ok = yield from self.wait(lambda: self.empty >= n)
                if not ok:
                    return
            self.item = n
            yield
            self.full += 1  # (the copies land, or the end is told)
            if n:
                ok = yield from self.wait(lambda: self.stored >= n)
                if not ok:
                    return

    def warp(self):
        n = 0
        while True:
            landed = yield from self.wait(lambda: self.full > n)
            item = self.item if landed else 0
            if not self.agree and not landed:
                item = self.item
            if not landed:
                self.lost = n if self.named else -1
            if item >= self.items:
                if self.agree:
                    for _ in range(SWEEPS):
                        yield from self.barrier()
                return
            yield
            self.n_empty += 1
            if self.n_empty == WARPS:
                self.n_empty, self.empty = 0, self.empty + 1
            for _ in range(SWEEPS):
                yield
                yield from self.barrier()
            if self.lost is not None and self.lost <= n:
                return
            assert landed and item == n
            self.stores[item] += 1
            yield
            self.n_stored += 1
            if self.n_stored == WARPS:
                self.n_stored, self.stored = 0, self.stored + 1
            n += 1

    def run(self):
        first = self.producer()
        live = [first] + [self.warp() for _ in range(WARPS)]
        slow = self.rng.choice((0.0, 0.9, 0.99))  # (how often the producer is held up)
        stuck = 0
        while live:
            self.clock += 1
            t = self.rng.choice(live)
            if t is first and len(live) > 1 and self.rng.random() < slow:
                continue
            try:
                stuck = stuck + 1 if next(t) == "barrier" else 0
            except StopIteration:
                live.remove(t)
                stuck = 0
            if stuck > 4000:  # everybody who is left waits in a barrier
                return False
            if self.clock > 100000:  # (a producer that left: the warps' limits)
                self.impatient = True
        assert all(x in (0, WARPS) for x in self.stores)
        assert self.impatient or self.stores[:-1] == [WARPS] * self.items
        return True


@pytest.mark.parametrize("items", [1, 2, 5])
def test_no_warp_is_left_in_a_barrier(items):
    for seed in range(150):
        assert Block(items, random.Random(seed)).run(), seed


def test_the_model_sees_the_warps_disagree():
    """A warp that leaves without the barriers; a mark that a slower warp takes
    for its own item's."""
    assert not all(Block(2, random.Random(seed), agree=False).run() for seed in range(1000))
    assert not all(Block(5, random.Random(seed), named=False).run() for seed in range(400))
