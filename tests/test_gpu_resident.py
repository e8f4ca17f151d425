"""The resident Jacobi solve (k_jacobi_res) where it can go wrong: one region
and just more than one along either axis, last regions of a few rows or
columns, sweep counts around whole phases, each of its forms (regions of 4, 8
and 12 warps, two regions an SM), weights other than 1, and a region that
stops sending."""
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


@pytest.mark.parametrize("w,h,iters,omega,tb", [
    (30, 126, 8, 1.0, 8), (31, 127, 9, 1.0, 8), (46, 238, 16, 1.0, 4), (47, 239, 17, 0.9, 8),
    (15, 353, 1, 1.0, 8), (260, 20, 40, 1.0, 3), (514, 130, 25, 0.8, 8),
    (700, 500, 23, 1.0, 8), (1024, 768, 17, 1.0, 5), (1200, 1250, 16, 1.0, 8),
])
def test_resident_solve_bitwise(gpu, w, h, iters, omega, tb):
    from oracle.pyoracle import OracleFluid

    p = dict(scheme=1, num_iters=iters, early_exit=False, jacobi_omega=omega)
    g = gpu.Fluid(1.0, w, h, 1.0, tb_depth=tb, **p)
    o = OracleFluid(1.0, w, h, 1.0, prec=32, threads=8, check_every=tb, **p)
    rng = np.random.default_rng(w + h)
    S = (rng.random(g.numCells) > 0.04).astype(np.float32)
    for f in (g, o):
        f.S[:] = S
        scenes.random_state(f, seed=iters, amp=1.0)
    for _ in range(2):  # (the second solve's packets meet the first one's)
        for f in (g, o):
            f.makeIncompressible(iters, 0.1)
    for k in ("U", "V", "p"):
        a, b = getattr(g, k), getattr(o, k)
        bad = a.view(np.uint32) != b.view(np.uint32)
        assert not bad.any(), (w, h, k, int(bad.sum()))
    assert g.stats()["sweeps"] == iters


def test_stalled_region_times_out_and_handle_recovers(gpu):
    from fluid_gb300 import _lib

    p = dict(scheme=1, num_iters=24, early_exit=False)
    a, b = (gpu.Fluid(1.0, 128, 128, 1.0, **p) for _ in range(2))
    for f in (a, b):
        scenes.fast_walls(f)
        scenes.random_state(f, seed=8, amp=0.5)
    start = {k: getattr(a, k).copy() for k in ("U", "V", "M", "newU", "newV", "newM")}
    a.debug_stall_tile(5)
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
    for k in ("U", "V", "M", "p"):
        x, y = getattr(a, k), getattr(b, k)
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), k


def test_batch_in_several_resident_launches_bitwise(gpu):
    """More scenes than one launch holds, sizes from one region to many."""
    sides = [62, 63, 64, 130, 200, 500, 512, 480, 300, 90, 70, 450, 410, 505, 260, 350, 500, 490]
    def make():
        out = []
        for n, s in enumerate(sides):
            f = gpu.Fluid(1.0, s, s + n, 1.0, auto_sync=False, scheme=1, num_iters=20 + 7 * n,
                          early_exit=False)
            scenes.ensemble_scene(f, np.random.default_rng(n))
            r = np.random.default_rng(100 + n)
            f.U[:] = r.uniform(-1, 1, f.numCells)
            f.V[:] = r.uniform(-1, 1, f.numCells)
            f.mark_dirty()
            out.append(f)
        return out
    alone, members = make(), make()
    batch = gpu.Batch(members)
    for _ in range(3):
        batch.step(0.1)
        for f in alone:
            f.Simulate(0.1)
    batch.scatter()
    for n, (a, m) in enumerate(zip(alone, members)):
        a.download()
        m.download()
        for k in ("U", "V", "M", "p"):
            x, y = getattr(a, k), getattr(m, k)
            assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), (n, k)
