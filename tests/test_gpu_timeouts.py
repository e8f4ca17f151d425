"""A bounded device-side wait that gives up is reported wherever a caller can
notice it: by a batch's scatter, losses and gradients, and by a recorded
rollout's loss and gradients.  The wait is made to run out by a region that
sends nothing (about a second a solve); the handle works again afterwards."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gpu():
    import fluid_gb300

    fluid_gb300.build()
    return fluid_gb300


def members(gpu, n=3):
    out = []
    for k in range(n):
        f = gpu.Fluid(1.0, 480, 480, 1.0, auto_sync=False, scheme=1, num_iters=24,
                      early_exit=False)
        scenes.ensemble_scene(f, np.random.default_rng(k))
        f.download()  # (queued edits reach the device)
        out.append(f)
    return out


def fields(fs):
    out = []
    for f in fs:
        f.download()
        out += [getattr(f, k).copy() for k in ("U", "V", "M", "p")]
    return out


def same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in zip(a, b))


def timed_out(gpu, call):
    from fluid_gb300 import _lib

    with pytest.raises(gpu.FluidError) as e:
        call()
    assert e.value.code == _lib.FG_ERR_TIMEOUT


def test_batch_reports_and_recovers(gpu):
    fs, ref = members(gpu), members(gpu)
    start = fields(fs)
    b = gpu.Batch(fs)
    b.debug_stall_tile(7)
    b.step(0.05)
    b.debug_stall_tile(-1)
    b.step(0.05)  # (a later step does not wipe the mark)
    timed_out(gpu, b.scatter)
    assert same(fields(fs), start)  # the members kept their state
    timed_out(gpu, b.scatter)
    b.gather()
    b.step(0.05)
    b.scatter()
    for f in ref:
        f.Simulate(0.05)
    assert same(fields(fs), fields(ref))


def test_batch_rollout_reports(gpu):
    fs = members(gpu)
    targets = [scenes.gaussian_target(f.NumX, f.NumY, seed=k) for k, f in enumerate(fs)]
    b = gpu.Batch(fs)
    b.debug_stall_tile(3)
    b.tape_begin(1)
    b.step_forward(0.05)
    timed_out(gpu, lambda: b.seed_smoke_l2(targets))
    b.step_adjoint()
    for s in range(3):
        timed_out(gpu, lambda: b.grad(s))
    b.tape_end()
    b.debug_stall_tile(-1)
    b.gather()
    losses, grads = b.rollout_grad(0.05, 1, targets)
    assert np.isfinite(losses).all() and len(grads) == 3


def test_rollout_reports(gpu):
    f = gpu.Fluid(1.0, 128, 128, 1.0, auto_sync=False, scheme=1, num_iters=24, early_exit=False)
    scenes.ensemble_scene(f, np.random.default_rng(1))
    target = scenes.gaussian_target(f.NumX, f.NumY, seed=1)
    f.download()
    start = {k: getattr(f, k).copy() for k in gpu.FIELDS}
    want = f.rollout_grad(0.05, 2, target)
    f.debug_stall_tile(5)
    timed_out(gpu, lambda: f.rollout_grad(0.05, 1, target))  # (at the loss)
    f.tape_begin(1)
    f.step_forward(0.05)
    timed_out(gpu, f.stats)
    f.tape_seed(dM=target)
    f.step_adjoint()
    timed_out(gpu, f.tape_grad)
    f.tape_end()
    f.debug_stall_tile(-1)
    f.download()
    for k, v in start.items():
        getattr(f, k)[:] = v
    f.mark_dirty()
    got = f.rollout_grad(0.05, 2, target)
    assert got["loss"] == want["loss"]
    for k in ("U", "V", "M"):
        assert np.linalg.norm(got[k] - want[k]) <= 1e-4 * np.linalg.norm(want[k])
