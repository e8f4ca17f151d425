"""The resident Jacobi solve's buffers are optional: where they cannot be
allocated a handle and a batch are made all the same, and their solves run in
the other kernels with the same result; grids that no form takes hold none."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import fluid_gb300

    fluid_gb300.build()
    return fluid_gb300


def first_made(gpu, make):
    """The first object made with one allocation failing, and how many failed
    the making before it."""
    for n in range(100):
        gpu.debug_fail_alloc(n)
        try:
            return make(), n
        except gpu.FluidError:
            continue
        finally:
            gpu.debug_fail_alloc(-1)
    raise AssertionError("never made")


def scene(f, seed):
    scenes.ensemble_scene(f, np.random.default_rng(seed))
    return f


def same(a, b):
    for k in ("U", "V", "M", "p"):
        x, y = getattr(a, k), getattr(b, k)
        assert np.array_equal(x.view(np.uint32), y.view(np.uint32)), k


@pytest.mark.parametrize("w,h", [(64, 64), (70, 65), (333, 222), (480, 480)])
def test_handle_without_the_buffers(gpu, w, h):
    make = lambda: gpu.Fluid(1.0, w, h, 1.0, auto_sync=False, scheme=1, num_iters=30,
                             early_exit=False)
    a, failed = first_made(gpu, make)
    b = make()
    assert failed > 20
    for f in (a, b):
        scene(f, w)
        for _ in range(2):
            f.Simulate(0.05)
    assert a.stats()["jacobi_resident"] == 0 and b.stats()["jacobi_resident"] > 0
    a.download()
    b.download()
    same(a, b)


def test_batch_without_the_buffers(gpu):
    make = lambda: [scene(gpu.Fluid(1.0, 480, 480, 1.0, auto_sync=False, scheme=1, num_iters=30,
                                    early_exit=False, use_graphs=0), n) for n in range(3)]
    members, alone = make(), make()
    for m in members:
        m.download()  # (edits and mirrors reach the device before an allocation may fail)
    batch, _ = first_made(gpu, lambda: gpu.Batch(members))
    full = gpu.Batch(alone)
    counts = []
    for b in (batch, full):
        n0 = b.launch_count()
        b.step(0.05)
        b.synchronize()
        counts.append(b.launch_count() - n0)
        b.scatter()
    assert counts[0] - counts[1] == 4 - 1  # four launches of 8 sweeps for the one
    for a, m in zip(alone, members):
        a.download()
        m.download()
        same(a, m)


def test_grids_of_no_form_hold_no_buffers(gpu):
    """The device memory of a 2046 x 2046 handle is its fields' and scratch's:
    5 bytes a cell for flags and mask beside 4 a float field, with nothing like
    the 19 MB that a form of 494 regions would take."""
    import torch

    free = lambda: (torch.cuda.synchronize(), torch.cuda.mem_get_info()[0])[1]
    make = lambda: gpu.Fluid(1.0, 2046, 2046, 1.0, auto_sync=False, scheme=1)
    make()
    f0 = free()
    f = make()
    used = f0 - free()
    fields = 8 + 3 + 17  # state, rotation partners, scratch
    floats = f.NumX * f.NumY * (fields + 2)  # + the noise table's pairs
    assert used < 4 * floats + f.NumX * f.NumY + (14 << 20), used
