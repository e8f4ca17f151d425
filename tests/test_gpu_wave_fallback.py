"""The serial schemes on one block, which is what runs when the pipeline's
buffers cannot be allocated (an injected failure at the first step): the SOR
with a fixed sweep count and with the early exit, and the reference's V-cycle
(its smoothers, its stop latch and the coarse Gauss-Seidel) on even and odd
sides, bit for bit against the oracle."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,p", [
    (60, 41, dict(num_iters=30, early_exit=False)),
    (201, 90, dict(num_iters=1, early_exit=False)),
    (64, 64, dict(num_iters=60, tolerance=1e-3)),
    (62, 62, dict(num_iters=3, UseMultigrid=True)),
    (97, 64, dict(num_iters=2, UseMultigrid=True)),
    (40, 133, dict(num_iters=2, UseMultigrid=True, PressureDamping=0.9)),
    (31, 33, dict(num_iters=30, UseMultigrid=True, tolerance=0.05)),
])
def test_one_block_schemes_bitwise(w, h, p):
    import fluid_gb300
    from oracle.pyoracle import OracleFluid

    fluid_gb300.build()
    g = fluid_gb300.Fluid(1.0, w, h, 1.0, UseBFECC=True, **p)
    o = OracleFluid(1.0, w, h, 1.0, prec=32, UseBFECC=True, **p)
    for f in (g, o):
        scenes.jet_scene(f)
        scenes.random_state(f, seed=w, amp=0.5)
    g.mark_dirty()
    g.download()  # (queued edits and mirrors reach the device first)
    fluid_gb300.debug_fail_alloc(0)
    try:
        g.Simulate(0.1)
    finally:
        fluid_gb300.debug_fail_alloc(-1)
    o.Simulate(0.1)
    for k in ("U", "V", "M", "p"):
        a, b = getattr(g, k), getattr(o, k)
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), k
    assert g.stats()["sweeps"] == o.stats()["sweeps"]
