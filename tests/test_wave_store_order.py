"""The order of a warp's shared-memory stores in k_wave's SOR sweep
(fluid_gb300/csrc/k_lexsor.cu).  Within a chunk of 16 steps the lanes are kept
together by shuffles, which order no memory: between two barriers of the warp
the stores of different lanes may become visible in any order, each lane's own
in the order it made them.  The model makes one sweep over a strip of 32 rows
chunk by chunk, applies a chunk's stores in random interleavings of the lanes
and compares the ring's U with the serial loop."""
import os
import random

import numpy as np
import pytest

C, LANES = 16, 32


def serial(U, V, rel):
    rows, NY = V.shape
    U, V = U.copy(), V.copy()
    for i in range(rows):
        for j in range(NY - 1):
            pp = -(U[i + 1, j] - U[i, j] + V[i, j + 1] - V[i, j]) / 4 * rel
            U[i, j] -= pp
            U[i + 1, j] += pp
            V[i, j] -= pp
            V[i, j + 1] += pp
    return U, V


def sweep(U, V, rel, rng, east):
    """east: the lanes that store their cell's east face."""
    NY = V.shape[1]
    U, V = U.copy(), V.copy()
    sent = np.zeros(LANES)  # the shuffles' values: each lane's last east face
    vcar = V[:, 0].copy()
    for s0 in range(0, NY + LANES, C):
        queue = [[] for _ in range(LANES)]
        for s in range(s0, s0 + C):
            new = sent.copy()
            for l in range(LANES):
                j = s - l
                if not 0 <= j < NY - 1:
                    continue
                # (Column 0's west value and lane 0's come from the ring; the
                # lane above has not reached column j yet.)
                west = U[0, j] if l == 0 else sent[l - 1]
                en, tn = U[l + 1, j], V[l, j + 1]
                pp = -(en - west + tn - vcar[l]) / 4 * rel
                queue[l].append(("U", l, j, west - pp))
                if l in east:
                    queue[l].append(("U", l + 1, j, en + pp))
                queue[l].append(("V", l, j, vcar[l] - pp))
                new[l] = en + pp
                vcar[l] = tn + pp
                if j == NY - 2:
                    queue[l].append(("V", l, j + 1, vcar[l]))
            sent = new
        todo = [l for l in range(LANES) for _ in queue[l]]
        rng.shuffle(todo)
        at = [0] * LANES
        for l in todo:
            f, i, j, x = queue[l][at[l]]
            at[l] += 1
            (U if f == "U" else V)[i, j] = x
    return U, V


def fields(NY, seed):
    r = np.random.default_rng(seed)
    return r.uniform(-1, 1, (LANES + 1, NY)), r.uniform(-1, 1, (LANES, NY))


@pytest.mark.parametrize("NY", [2, 17, 40, 97])
def test_stores_of_a_chunk_may_land_in_any_order(NY):
    U, V = fields(NY, NY)
    want = serial(U, V, 1.7)
    for seed in range(20):
        got = sweep(U, V, 1.7, random.Random(seed), {LANES - 1})
        assert all(np.array_equal(a, b) for a, b in zip(got, want)), seed


def test_the_model_sees_two_lanes_storing_one_word():
    U, V = fields(40, 1)
    want = serial(U, V, 1.7)
    got = sweep(U, V, 1.7, random.Random(0), set(range(LANES)))
    assert not np.array_equal(got[0], want[0])


def test_the_kernel_stores_the_last_lanes_east_face_only():
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    text = open(os.path.join(root, "fluid_gb300", "csrc", "k_lexsor.cu")).read()
    stores = [x.strip() for x in text.splitlines() if "F(at0 + RB) = en" in x]
    assert stores == ["if (lane == 31) F(at0 + RB) = en;"]
