"""Which kernel ran a Jacobi solve: the resident launch in each of its forms
(regions of 4, 8 and 12 warps, two regions of 8 warps an SM), the launches and
the dataflow kernel on grids beyond its capacity, and the launches of a batch.
fg_stats names them, and every result equals the oracle's bit for bit, so a
kernel that silently stops running fails here."""
import os
import subprocess
import sys

import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def gpu():
    import fluid_gb300

    fluid_gb300.build()
    return fluid_gb300


def solve(gpu, w, h, iters, **kw):
    from oracle.pyoracle import OracleFluid

    p = dict(scheme=1, num_iters=iters, early_exit=kw.pop("early_exit", False))
    tb = kw.pop("tb_depth", 8)
    g = gpu.Fluid(1.0, w, h, 1.0, tb_depth=tb, **p, **kw)
    o = OracleFluid(1.0, w, h, 1.0, prec=32, threads=8, check_every=tb, **p, **kw)
    S = (np.random.default_rng(w + h).random(g.numCells) > 0.04).astype(np.float32)
    for f in (g, o):
        f.S[:] = S
        scenes.random_state(f, seed=iters, amp=1.0)
        f.makeIncompressible(iters, 0.1)
    for k in ("U", "V", "p"):
        a, b = getattr(g, k), getattr(o, k)
        bad = a.view(np.uint32) != b.view(np.uint32)
        assert not bad.any(), (w, h, k, int(bad.sum()))
    st = g.stats()
    assert st["sweeps"] == o.stats()["sweeps"]
    return st["jacobi_resident"], st["jacobi_kernel"]


@pytest.mark.parametrize("w,h,iters,tb,form", [
    (62, 62, 24, 8, 4), (128, 128, 24, 8, 4), (270, 126, 24, 8, 4),
    (271, 126, 24, 8, 8), (192, 192, 24, 8, 8), (512, 256, 24, 8, 8), (700, 500, 23, 8, 8), (1024, 768, 17, 5, 12), (400, 2700, 12, 4, 12),
    (1200, 800, 24, 8, 12), (1200, 1250, 16, 8, 16),
])
def test_resident_forms(gpu, w, h, iters, tb, form):
    assert solve(gpu, w, h, iters, tb_depth=tb)[0] == form


@pytest.mark.parametrize("w,h,iters,kw,kernel", [
    (9000, 260, 24, {}, "DATAFLOW"), (600, 4000, 40, {}, "DATAFLOW"),  # 339 and 288 tiles
    (30000, 100, 16, {}, "DATAFLOW"),                 # one tile column
    (900, 2700, 12, dict(tb_depth=4), "SWEEP"),       # depths below 8
    (9000, 260, 8, {}, "TMA"),                        # one full launch
    (333, 222, 40, dict(early_exit=True, tolerance=0.0), "SWEEP"),
    (70, 45, 40, dict(early_exit=True, tolerance=1e-2), "SWEEP"),
])
def test_solves_that_are_not_resident(gpu, w, h, iters, kw, kernel):
    assert solve(gpu, w, h, iters, **kw) == (0, getattr(gpu, "JACOBI_KERNEL_" + kernel))


FRESH = r"""
import sys
sys.path.insert(0, sys.argv[1])
import fluid_gb300 as fg
f = fg.Fluid(1.0, 1100, 1500, 1.0, auto_sync=False, scheme=1, num_iters=40, tb_depth=8,
             early_exit=False)
S = f.S.reshape(f.NumX, f.NumY)
S[:] = 1.0
S[:, 0] = S[:, -1] = S[0, :] = 0.0
f.mark_dirty()
for _ in range(3):
    f.Simulate(0.1)
    st = f.stats()
    assert (st["jacobi_resident"], st["jacobi_kernel"]) == (0, fg.JACOBI_KERNEL_DATAFLOW), st
"""


def test_dataflow_kernel_in_the_graph_of_a_fresh_process():
    """No CUDA call before the handle: its captured steps hold the dataflow
    kernel on a grid that the resident launch does not take."""
    subprocess.run([sys.executable, "-c", FRESH, ROOT], check=True, timeout=300)


def test_batch_runs_resident_launches(gpu):
    """A batch of 150 regions, which the plan solves in one launch a step
    whatever its sweeps (in launches of 8, four times the sweeps take more)."""
    counts = []
    for more in (1, 4):
        fs = []
        for n, s in enumerate((480, 480, 480)):
            f = gpu.Fluid(1.0, s, s, 1.0, auto_sync=False, scheme=1,
                          num_iters=(40 + 16 * n) * more, early_exit=False, use_graphs=0)
            scenes.ensemble_scene(f, np.random.default_rng(n))
            fs.append(f)
        b = gpu.Batch(fs)
        n0 = b.launch_count()
        b.step(0.05)
        b.synchronize()
        counts.append(b.launch_count() - n0)
        b.close()
    assert counts[0] == counts[1] > 0
