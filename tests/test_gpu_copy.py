"""The list copy kernel (k_copy_list) where it can go wrong: widths that are
and are not multiples of 4, element counts with a remainder of 1 to 3, sizes
around the line between it and the copy engine, one field and all of them, and
batches of more slices than one launch takes.  Each value goes from the host
mirror to its handle, to the batch's packed field, back, and to the mirror."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STEP_FIELDS = ("U", "V", "M", "p", "newU", "newV", "newM")


def round_trip(sizes):
    import fluid_gb300 as gpu

    p = dict(scheme=gpu.SCHEME_JACOBI, num_iters=8, early_exit=False, auto_sync=False)
    fs = [gpu.Fluid(1.0, w, h, 1.0, **p) for w, h in sizes]
    want = []
    for n, f in enumerate(fs):
        rng = np.random.default_rng(n)
        f.S[:] = rng.integers(0, 2, f.numCells)
        for k in STEP_FIELDS:
            getattr(f, k)[:] = rng.standard_normal(f.numCells).astype(np.float32)
        want.append({k: getattr(f, k).copy() for k in STEP_FIELDS})
        f.mark_dirty()
    b = gpu.Batch(fs)
    for f in fs:
        for k in STEP_FIELDS:
            getattr(f, k)[:] = -1.0
    b.scatter()
    for f, w in zip(fs, want):
        f.download(1 << gpu.FIELDS["V"])
        assert np.array_equal(f.V, w["V"]), (f.NumX, f.NumY)
        assert (f.U == -1.0).all()
        f.download()
        for k in STEP_FIELDS:
            assert np.array_equal(getattr(f, k), w[k]), (f.NumX, f.NumY, k)
    b.close()


@pytest.mark.parametrize("w,h", [(1, 1), (2, 2), (3, 5), (1, 29), (1, 31), (30, 33), (5, 98), (128, 128),
                                 (300, 251), (360, 410), (390, 397), (700, 801), (1020, 1030)])
def test_copies_keep_every_value(w, h):
    round_trip([(w, h)])


def test_copies_of_many_scenes():
    round_trip([(8 + 3 * k, 40 - k) for k in range(39)])


@pytest.mark.parametrize("counts", [(1, 2, 3), (5, 16384, 7), (16385, 3), (3, 16383)])
def test_particles_come_back_in_order(counts):
    import fluid_gb300 as gpu

    f = gpu.Fluid(1.0, 40, 30, 1.0, auto_sync=False)
    rng = np.random.default_rng(7)
    want = {k: np.zeros(0, np.float32) for k in ("X", "Y", "MaxAge")}
    rgb = np.zeros((0, 3), np.uint8)
    assert f.particles()["X"].size == 0
    for n in counts:
        x, y, age = (rng.uniform(1, 30, n).astype(np.float32) for _ in range(3))
        c = rng.integers(0, 256, (n, 3)).astype(np.uint8)
        f.particles_add(x, y, age, c)
        for k, v in zip(("X", "Y", "MaxAge"), (x, y, age)):
            want[k] = np.concatenate([want[k], v])
        rgb = np.concatenate([rgb, c])
        got = f.particles()
        for k, v in want.items():
            assert np.array_equal(got[k], v), (n, k)
        assert not got["Age"].any() and np.array_equal(got["RGB"], rgb)
    f.particles_clear()
    assert f.particles()["X"].size == 0
    f.particles_add(x[:3], y[:3], age[:3], c[:3])
    assert np.array_equal(f.particles()["Y"], y[:3])


@pytest.mark.parametrize("w,h", [(1, 1), (31, 40), (510, 1030), (2100, 2046)])
def test_view_ranges(w, h):
    """The one-block and the two-level reductions of a view's range."""
    import fluid_gb300 as gpu

    f = gpu.Fluid(1.0, w, h, 1.0, auto_sync=False)
    f.S[:] = 1
    f.M[:] = np.random.default_rng(1).uniform(-3, 5, f.numCells).astype(np.float32)
    f.U[:] = 2 * f.M
    f.V[:] = 0.5 - f.M
    f.mark_dirty()
    v = f.Smoke()
    assert (v.MinValue, v.MaxValue) == (f.M.min(), f.M.max())
    for v in (f.Vorticity(), f.VelocityMagnitude()):
        inner = v.values.reshape(f.NumX, f.NumY)[1:-1, 1:-1]
        assert (v.MinValue, v.MaxValue) == (inner.min(), inner.max())
