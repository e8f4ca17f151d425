"""The serial schemes' pipeline (k_wave) at the sizes where it can go wrong:
strip and group remainders, columns around the ring's wrap, more sweeps than
one launch takes, values small enough to divide in the subnormal range, and a
strip that stops sending."""
import time

import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import fluid_gb300

    fluid_gb300.build()
    return fluid_gb300


def pair(gpu, w, h, **params):
    from oracle.pyoracle import OracleFluid

    return (gpu.Fluid(1.0, w, h, 1.0, **params), OracleFluid(1.0, w, h, 1.0, prec=32, **params))


def same(g, o, fields=("U", "V", "p"), where=""):
    for k in fields:
        a, b = getattr(g, k), getattr(o, k)
        bad = a.view(np.uint32) != b.view(np.uint32)
        assert not bad.any(), (where, k, int(bad.sum()))


@pytest.mark.parametrize("w,h,iters,early", [
    (23, 30, 8, False), (24, 31, 8, True), (25, 222, 9, False), (30, 223, 1, True),
    (31, 224, 2, False), (56, 254, 7, True), (57, 255, 17, False), (64, 285, 16, True),
    (300, 6, 40, False), (3, 700, 24, True), (2, 2, 5, False),
])
def test_strip_and_ring_edges_bitwise(gpu, w, h, iters, early):
    g, o = pair(gpu, w, h, num_iters=iters, early_exit=early, tolerance=0.02, PressureDamping=0.97)
    rng = np.random.default_rng(w * 1000 + h)
    S = (rng.random(g.numCells) > 0.06).astype(np.float32)
    for f in (g, o):
        f.S[:] = S
        scenes.random_state(f, seed=iters, amp=1.0)
        f.makeIncompressible(iters, 0.1)
    same(g, o, where="%dx%d" % (w, h))
    assert g.stats()["sweeps"] == o.stats()["sweeps"]
    assert g.stats()["last_maxdiv"] == o.stats()["last_maxdiv"]


def test_subnormal_and_zero_quotients_bitwise(gpu):
    """Velocities down to the subnormal range beside walls (three fluid
    neighbours: the division by 3) and exact zeros of both signs."""
    g, o = pair(gpu, 70, 61)
    rng = np.random.default_rng(3)
    n = g.numCells
    mag = np.ldexp(rng.uniform(-1, 1, (2, n)), rng.integers(-150, 0, (2, n))).astype(np.float32)
    mag[rng.random((2, n)) < 0.2] = -0.0
    S = (rng.random(n) > 0.3).astype(np.float32)
    for f in (g, o):
        f.S[:] = S
        f.U[:], f.V[:] = mag
        f.makeIncompressible(3, 0.1)
    same(g, o)


@pytest.mark.parametrize("tol", [0.0, 2e-6])
def test_more_sweeps_than_one_launch_bitwise(gpu, tol):
    g, o = pair(gpu, 20, 37, num_iters=2100, tolerance=tol)
    for f in (g, o):
        f.S[:] = 1.0
        f.S[: f.NumY] = 0.0
        scenes.random_state(f, seed=4, amp=1.0)
        f.makeIncompressible(2100, 0.1)
    same(g, o)
    assert g.stats()["sweeps"] == o.stats()["sweeps"]


@pytest.mark.parametrize("w,h", [(45, 470), (470, 45), (129, 258)])
def test_reference_vcycle_edges_bitwise(gpu, w, h):
    g, o = pair(gpu, w, h, UseMultigrid=True, num_iters=3)
    for f in (g, o):
        scenes.fast_walls(f)
        scenes.random_state(f, seed=6, amp=0.5)
        f.makeIncompressible(3, 0.1)
    same(g, o)


def test_stalled_strip_times_out_and_handle_recovers(gpu):
    from fluid_gb300 import _lib

    a, b = (gpu.Fluid(1.0, 100, 60, 1.0) for _ in range(2))
    for f in (a, b):
        scenes.fast_walls(f)
        scenes.random_state(f, seed=8, amp=0.5)
    start = {k: getattr(a, k).copy() for k in ("U", "V", "M", "newU", "newV", "newM")}
    a.debug_stall_tile(1)
    t0 = time.monotonic()
    a.Simulate(0.1)
    with pytest.raises(gpu.FluidError) as e:
        a.stats()
    assert e.value.code == _lib.FG_ERR_TIMEOUT
    assert time.monotonic() - t0 < 30.0
    a.debug_stall_tile(-1)
    for k, v in start.items():
        getattr(a, k)[:] = v
    for f in (a, b):
        f.Simulate(0.1)
        f.stats()
    same(a, b, fields=("U", "V", "M", "p"))
