"""A host model of the serial schemes' pipeline (k_wave in
fluid_gb300/csrc/k_lexsor.cu): strips of 32 rows, one warp per sweep marching
along the columns in chunks, the ring of columns in shared memory, the packets
between strips, the ticket order of the tasks.  The warps run step by step
under random interleavings with every index checked against its buffer; each
value must come out as the serial loop's, bit for bit in float64, and nothing
may deadlock."""
import random

import numpy as np
import pytest

G8, C, W = 8, 16, 256  # WV_G, WV_C, WV_W
LANE = np.arange(32)


def serial(U, V, p, S, sweeps, rel):
    NX, NY = S.shape
    for t in range(sweeps):
        for i in range(1, NX - 1):
            for j in range(1, NY - 1):
                if not S[i, j]:
                    continue
                n = (S[i - 1, j], S[i + 1, j], S[i, j - 1], S[i, j + 1])
                s = sum(n)
                if not s:
                    continue
                pp = -(U[i + 1, j] - U[i, j] + V[i, j + 1] - V[i, j]) / s * rel[t]
                p[i, j] += 0.7 * pp
                U[i, j] -= n[0] * pp
                U[i + 1, j] += n[1] * pp
                V[i, j] -= n[2] * pp
                V[i, j + 1] += n[3] * pp


def serial_gs(P, R, S, sweeps, rel):
    NX, NY = S.shape
    for _ in range(sweeps):
        for i in range(1, NX - 1):
            for j in range(1, NY - 1):
                n = (S[i - 1, j], S[i + 1, j], S[i, j - 1], S[i, j + 1])
                if not S[i, j] or not sum(n):
                    continue
                x = P[i, j]
                lap = (n[0] * (P[i - 1, j] - x) + n[1] * (P[i + 1, j] - x) + n[2] * (P[i, j - 1] - x) +
                       n[3] * (P[i, j + 1] - x))
                P[i, j] = x + -(R[i, j] - lap) / sum(n) * rel


class Model:
    def __init__(self, gs, fields, S, sweeps, rel, blocks, rng):
        self.gs, self.S, self.sweeps, self.rel, self.rng = gs, S, sweeps, rel, rng
        self.NX, self.NY = S.shape
        self.P = -(-self.NY // 32) * 32
        self.dst = [np.pad(f, ((0, 0), (0, self.P - self.NY)), constant_values=np.nan) for f in fields]
        self.G = min(G8, sweeps)
        self.B = (self.NX + self.G - 2 + 31) // 32
        self.ng = -(-sweeps // self.G)
        self.pkt, self.fin = {}, {}
        self.tasks = sorted(((b, g) for b in range(self.B) for g in range(self.ng)),
                            key=lambda x: (x[0] + 2 * x[1], x[1]))
        # The ticket decoding of the kernel gives the same order.
        key = before = 0
        for tk, want in enumerate(self.tasks):
            while True:
                g0, g1 = max(0, int((key - self.B + 2) / 2)), min(self.ng - 1, key // 2)
                if tk < before + g1 - g0 + 1:
                    g = g0 + tk - before
                    assert (key - 2 * g, g) == want
                    break
                before += max(g1 - g0 + 1, 0)
                key += 1
        self.blocks = blocks

    def flags(self, i, j):
        """(active, W, E, S, N) of a cell; all zero off the interior."""
        if not (1 <= i < self.NX - 1 and 1 <= j < self.NY - 1) or not self.S[i, j]:
            return (0, 0, 0, 0, 0)
        n = (self.S[i - 1, j], self.S[i + 1, j], self.S[i, j - 1], self.S[i, j + 1])
        return (1 if sum(n) else 0, *n)

    def task(self, b, g):
        gs, G, NY, P = self.gs, self.G, self.NY, self.P
        Gt = min(G, self.sweeps - g * G)
        nch = (NY + 31 - ((b & (C - 1)) - C) + 2 * Gt + C - 1) // C
        A = [np.full((33 + G8, W), np.nan), np.full((32 + G8, W), np.nan), np.full((32 + G8, W), np.nan)]
        F = np.full((32 + G8, W, 5), np.nan)
        before, past = 64, 96  # WV_BEFORE, WV_PAST
        F[:, W - before:] = 0.0
        st = dict(prog=[0] * G8, loaded=0, stored=0)
        i0 = 1 + 32 * b

        def rows(ring, src, q0, q1, c, data=True):
            for q in range(q0, q1):
                i = i0 + q - G8
                ring[q, (c & (W - 1)):(c & (W - 1)) + 32] = src[i, c:c + 32] if data and 0 <= i < self.NX else 0.0

        def loader():
            for c in range(0, P + past, 32):
                inside = min((32 - (((b & (C - 1)) - C)) + 2 * Gt + C - 1) // C, nch)
                while (c >= W and c + 32 - W > st["stored"]) or (
                        W - before <= c < W and inside > st["prog"][Gt - 1]):
                    yield False
                for d in (0, 1):
                    if g and b + d < self.B and c < P:
                        while self.fin.get((b + d, g - 1), 0) < min(c + 32, NY):
                            yield False
                lo, hi = G8 - (G - 1), G8 + 32
                if c >= P:
                    pass
                elif gs:
                    rows(A[0], self.dst[0], G8 if b else G8 - G, hi + 1, c, g > 0)
                    rows(A[1], self.dst[1], lo, hi, c)
                else:
                    rows(A[0], self.dst[0], G8, hi + 1, c)
                    rows(A[1], self.dst[1], G8, hi, c)
                    rows(A[2], self.dst[2], G8, hi, c)
                for q in range(lo, hi):
                    for k in range(32):
                        F[q, (c + k) & (W - 1)] = self.flags(i0 + q - G8, c + k)
                yield True
                st["loaded"] = c + 32

        def storer():
            for c in range(0, P, 32):
                while st["prog"][Gt - 1] < min((c + 63 - ((b & (C - 1)) - C) + 2 * Gt + C - 1) // C, nch):
                    yield False
                for fd in range(1 if gs else 3):
                    for r in range(32):
                        i, q = i0 - (Gt - 1) + r, G8 - (Gt - 1) + r
                        if (0 if gs else 1) <= i < self.NX:
                            n = min(32, NY - c)
                            self.dst[fd][i, c:c + n] = A[fd][q, (c & (W - 1)):(c & (W - 1)) + n]
                yield True
                self.fin[b, g] = c + 32
                st["stored"] = c + 32

        def sweep(w):
            q = G8 - w + LANE
            rel = self.rel[g * G + w] if not gs else self.rel
            v0, ue = np.zeros(32), np.zeros(32)
            slot = (g & 1) * G + w
            s = ((b & (C - 1)) - C) - 2 * (w + 1)
            n0 = (-1 - s) // C
            s += n0 * C

            def fetch(j):
                c, cn = j & (W - 1), (j + 1) & (W - 1)
                return (A[0][q + 1, c], A[0][q, cn] if gs else A[1][q, cn],
                        A[1][q, c] if gs else A[2][q, c], F[q, c])

            nxt = None
            for n in range(n0, nch):
                if w == 0:
                    while st["loaded"] < min(s + C + 2, P + past):
                        yield False
                else:
                    while st["prog"][w - 1] < n + 1:
                        yield False
                if b > 0:
                    for c in range(max(s, 0), min(s + C, NY)):
                        while self.pkt.get((b - 1, slot, c), (0, 0))[1] != g + 1:
                            yield False
                        x = self.pkt[b - 1, slot, c][0]
                        ql = G8 - w
                        if gs:
                            assert ql >= 1
                            A[0][ql - 1, c & (W - 1)] = x[0]
                        else:
                            A[0][ql, c & (W - 1)] = x[0]
                            if w + 1 < Gt:
                                assert ql >= 1
                                A[1][ql - 1, c & (W - 1)], A[2][ql - 1, c & (W - 1)] = x[1], x[2]
                if n == n0:
                    nxt = fetch(s - LANE)
                for k in range(C):
                    j = s + k - LANE
                    wv = np.concatenate([[A[0][q[0] - 1 if gs else q[0], j[0] & (W - 1)]], ue[:-1]])
                    x1, x2, x3, fl = nxt
                    nxt = fetch(j + 1)
                    act = fl[:, 0] != 0
                    cnt = np.where(act, fl[:, 1:].sum(axis=1), 1)
                    c = j & (W - 1)
                    with np.errstate(invalid="ignore"):
                        if gs:
                            lap = (fl[:, 1] * (wv - v0) + fl[:, 2] * (x1 - v0) + fl[:, 3] * (ue - v0) +
                                   fl[:, 4] * (x2 - v0))
                            out = np.where(act, v0 + -(x3 - lap) / cnt * rel, v0)
                            A[0][q, c] = out
                            ue, v0 = out, x2
                        else:
                            pp = -(x1 - wv + x2 - v0) / cnt * rel
                            un = np.where(act, wv - fl[:, 1] * pp, wv)
                            en = np.where(act, x1 + fl[:, 2] * pp, x1)
                            vn = np.where(act, v0 - fl[:, 3] * pp, v0)
                            tn = np.where(act, x2 + fl[:, 4] * pp, x2)
                            pn = np.where(act, x3 + 0.7 * pp, x3)
                            A[0][q, c] = un  # (then the east face; the lane above stores last)
                            A[0][q[31] + 1, c[31]] = en[31]
                            A[1][q, c], A[2][q, c] = vn, pn
                            ue, v0 = en, tn
                    yield True
                out = {}
                for cs in range(max(s - 31, 0), min(s - 31 + C, NY)):
                    q31, m = G8 - w + 31, cs & (W - 1)
                    out[cs] = (A[0][q31, m],) if gs else (A[0][q31 + 1, m], A[1][q31, m], A[2][q31, m])
                yield True
                st["prog"][w] = n + 1
                yield True
                if b + 1 < self.B:
                    for cs, x in out.items():
                        self.pkt[b, slot, cs] = (x, g + 1)
                s += C
                yield True

        return [loader(), storer()] + [sweep(w) for w in range(Gt)]

    def run(self):
        todo, running, idle = list(self.tasks), [], 0
        while todo or running:
            while todo and len(running) < self.blocks:
                running.append(self.task(*todo.pop(0)))
            blk = self.rng.choice(running)
            it = self.rng.choice(blk)
            moved = False
            for _ in range(self.rng.randint(1, 12)):
                try:
                    r = next(it)
                    moved = moved or r
                    if not r:
                        break
                except StopIteration:
                    blk.remove(it)
                    moved = True
                    break
            if not blk:
                running.remove(blk)
            idle = 0 if moved else idle + 1
            assert idle < 200000, "deadlock"
        return [d[:, :self.NY] for d in self.dst]


CASES = [(5, 9, 1, 1), (34, 40, 3, 2), (70, 61, 35, 3), (40, 300, 9, 2), (98, 33, 16, 1), (20, 560, 16, 1), (66, 222, 20, 2)]


def mask(rng, nx, ny):
    S = (rng.random((nx, ny)) > 0.08).astype(float)
    S[0] = 0.0
    S[:, 0] = 0.0
    return S


@pytest.mark.parametrize("nx,ny,sweeps,blocks", CASES)
def test_sor_pipeline_equals_the_serial_loop(nx, ny, sweeps, blocks):
    rng = np.random.default_rng(nx * ny)
    S = mask(rng, nx, ny)
    U, V, p = (rng.uniform(-1, 1, (nx, ny)) for _ in range(3))
    rel = [1.9 - 0.7 * t / sweeps for t in range(sweeps)]
    got = Model(False, (U, V, p), S, sweeps, rel, blocks, random.Random(nx)).run()
    want = [U.copy(), V.copy(), p.copy()]
    serial(*want, S, sweeps, rel)
    for a, x in zip(got, want):
        assert np.array_equal(a, x)


@pytest.mark.parametrize("nx,ny,sweeps,blocks", [c for c in CASES if c[2] % 8 != 1])
def test_coarse_pipeline_equals_the_serial_loop(nx, ny, sweeps, blocks):
    rng = np.random.default_rng(nx + ny)
    S = mask(rng, nx, ny)
    R = rng.uniform(-1, 1, (nx, ny))
    start = np.zeros((nx, ny))
    got = Model(True, (np.full((nx, ny), np.nan), R), S, sweeps, 1.6, blocks, random.Random(ny)).run()
    serial_gs(start, R, S, sweeps, 1.6)
    assert np.array_equal(got[0], start)
