"""A host model of the resident Jacobi solve (k_jacobi_res in
fluid_gb300/csrc/k_pressure.cu): the regions' packets (which cells of a region
go into which packet, where each halo item comes from) and the two slots by
phase parity, under random interleavings of the blocks.  Every index is
checked against its buffer, every packet's tag against the phase, and the
result against plain Jacobi sweeps, bit for bit in float64."""
import random

import numpy as np
import pytest

H, RT, JT, RJ = 8, 8, 4, 128
JP = (RT * JT + 2) // 3
JROWS = 2 * JP * 32


def spans(n, R):
    S = R - 2 * H
    return 1 if n <= R else -(-(n - R) // S) + 1


def window(t, n, R):
    a = t * (R - 2 * H)
    return (H if t else 0), (n - a if a + R >= n else R - H)


class Region:
    def __init__(self, rid, ty, tx, nty, ntx, NX, NY, NW, W, BW):
        R = NW * RT
        self.id, self.ntx, self.NW = rid, ntx, NW
        self.up, self.down, self.left, self.right = ty > 0, ty < nty - 1, tx > 0, tx < ntx - 1
        self.r0, self.c0 = ty * (R - 2 * H), tx * (RJ - 2 * H)
        self.rows, self.cols = window(ty, NX, R), window(tx, NY, RJ)
        self.w, self.bw = np.zeros((R, RJ)), np.zeros((R, RJ))
        a, b = min(R, NX - self.r0), min(RJ, NY - self.c0)
        self.w[:a, :b] = W[self.r0:self.r0 + a, self.c0:self.c0 + b]
        self.bw[:a, :b] = BW[self.r0:self.r0 + a, self.c0:self.c0 + b]
        self.x = np.zeros((R, RJ))

    def sweep(self):
        p = np.pad(self.x, 1)
        # (a shuffle at lane 0 or 31 returns the thread's own value)
        p[1:-1, 0], p[1:-1, -1] = self.x[:, JT - 1], self.x[:, RJ - JT]
        self.x = self.w * (p[:-2, 1:-1] + p[2:, 1:-1] + p[1:-1, :-2] + p[1:-1, 2:]) + self.bw

    def cells(self, warp, lane):
        """The 32 values of a thread, padded to whole packets."""
        v = self.x[warp * RT:(warp + 1) * RT, lane * JT:(lane + 1) * JT].ravel()
        return np.concatenate([v, np.zeros(3 * JP - len(v))])

    def publish(self, put, ph, N):
        NW, base = self.NW, (self.id * 2 + (ph & 1)) * N
        for warp in range(NW):
            for lane in range(32):
                v = self.cells(warp, lane)
                outs = []
                if warp == 1 and self.up:
                    outs.append([base + m * 32 + lane for m in range(JP)])
                if warp == NW - 2 and self.down:
                    outs.append([base + (JP + m) * 32 + lane for m in range(JP)])
                if lane in (2, 3) and self.left:
                    outs.append([base + JROWS + warp * JP * 2 + lane - 2 + 2 * m for m in range(JP)])
                if lane in (28, 29) and self.right:
                    outs.append([base + JROWS + (NW + warp) * JP * 2 + lane - 28 + 2 * m for m in range(JP)])
                for at in outs:
                    for m in range(JP):
                        put(at[m], v[3 * m:3 * m + 3], ph)

    def sources(self, N):
        NW = self.NW
        for k in range(N):
            if k < JROWS:
                side, rest = divmod(k, JP * 32)
                lane = rest & 31
                dx = -1 if lane < 2 and self.left else 1 if lane >= 30 and self.right else 0
                if self.down if side else self.up:
                    yield k, ((self.ntx if side else -self.ntx) + dx) * 2 * N + (1 - side) * JP * 32 + rest - 28 * dx
            else:
                c = k - JROWS
                side, wr = c // (NW * JP * 2), (c // (JP * 2)) % NW
                covered = (wr == 0 and self.up) or (wr == NW - 1 and self.down)
                if (self.right if side else self.left) and not covered:
                    yield k, (2 * N if side else -2 * N) + JROWS + (1 - side) * NW * JP * 2 + c - side * NW * JP * 2

    def receive(self, stage):
        NW = self.NW
        for warp in range(NW):
            above, below = warp == 0 and self.up, warp == NW - 1 and self.down
            for lane in range(32):
                lcol, rcol = lane < 2 and self.left, lane >= 30 and self.right
                if not (above or below or lcol or rcol):
                    continue
                row = above or below
                first = ((JP * 32 if below else 0) + lane if row else
                         JROWS + ((NW if rcol else 0) + warp) * JP * 2 + (lane - 30 if rcol else lane))
                step = 32 if row else 2
                v = np.concatenate([stage[first + m * step] for m in range(JP)])[:RT * JT]
                self.x[warp * RT:(warp + 1) * RT, lane * JT:(lane + 1) * JT] = v.reshape(RT, JT)


@pytest.mark.parametrize("NX,NY,NW,iters", [(40, 130, 4, 21), (33, 129, 4, 16), (130, 250, 8, 27),
                                            (66, 100, 8, 17), (20, 353, 4, 24), (30, 60, 8, 9)])
def test_resident_solve_equals_plain_sweeps(NX, NY, NW, iters):
    rng = np.random.default_rng(NX * NY)
    active = np.zeros((NX, NY))
    active[1:-1, 1:-1] = rng.random((NX - 2, NY - 2)) > 0.05
    W = active * rng.uniform(0.1, 0.3, (NX, NY))
    BW = active * rng.uniform(-1, 1, (NX, NY))
    want = np.zeros((NX, NY))
    for _ in range(iters):
        p = np.pad(want, 1)
        want = W * (p[:-2, 1:-1] + p[2:, 1:-1] + p[1:-1, :-2] + p[1:-1, 2:]) + BW
    nty, ntx = spans(NX, NW * RT), spans(NY, RJ)
    N = JROWS + 2 * NW * JP * 2
    regions = [Region(ty * ntx + tx, ty, tx, nty, ntx, NX, NY, NW, W, BW)
               for ty in range(nty) for tx in range(ntx)]
    size = len(regions) * 2 * N
    buf, tags = [None] * size, [-1] * size
    pick = random.Random(NX)

    def put(at, v, ph):
        assert 0 <= at < size
        buf[at], tags[at] = v.copy(), ph

    def run(r):
        nph = -(-iters // H)
        for ph in range(nph):
            for _ in range(min(H, iters - ph * H)):
                r.sweep()
            if ph + 1 == nph:
                return
            yield
            r.publish(put, ph, N)
            yield
            stage = {}
            own = (r.id * 2 + (ph & 1)) * N
            for k, at in r.sources(N):
                assert 0 <= own + at < size
                while tags[own + at] != ph:
                    assert tags[own + at] < ph, "overwritten before it was read"
                    yield
                stage[k] = buf[own + at]
            r.receive(stage)

    live = [run(r) for r in regions]
    for _ in range(10 ** 6):
        if not live:
            break
        it = pick.choice(live)
        try:
            next(it)
        except StopIteration:
            live.remove(it)
    assert not live, "deadlock"
    got = np.full((NX, NY), np.nan)
    for r in regions:
        a, b, c, d = *r.rows, *r.cols
        a1, d1 = min(b, NX - r.r0), min(d, NY - r.c0)
        got[r.r0 + a:r.r0 + a1, r.c0 + c:r.c0 + d1] = r.x[a:a1, c:d1]
    assert np.array_equal(got, want)
