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
