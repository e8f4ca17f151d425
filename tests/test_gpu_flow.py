"""The dataflow Jacobi kernel (k_jacobi_flow) at the edges of its 80 x 112
tiles: whole tiles along both axes, one row and column more, two tile rows of
which the second owns one, fewer and more than two tiles a block, a launch of
the remaining sweeps after it, and a weight other than 1."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,iters,omega", [
    (1438, 1230, 16, 1.0), (1439, 1231, 17, 1.0), (79, 17136, 24, 1.0),
    (1600, 1791, 24, 0.9), (1521, 2018, 40, 1.0),
])
def test_dataflow_solve_bitwise(w, h, iters, omega):
    import fluid_gb300
    from oracle.pyoracle import OracleFluid

    p = dict(scheme=1, num_iters=iters, early_exit=False, jacobi_omega=omega)
    g = fluid_gb300.Fluid(1.0, w, h, 1.0, **p)
    o = OracleFluid(1.0, w, h, 1.0, prec=32, threads=8, **p)
    rng = np.random.default_rng(w + h)
    S = (rng.random(g.numCells) > 0.04).astype(np.float32)
    for f in (g, o):
        f.S[:] = S
        scenes.random_state(f, seed=iters, amp=1.0)
        f.makeIncompressible(iters, 0.1)
    for k in ("U", "V", "p"):
        a, b = getattr(g, k), getattr(o, k)
        bad = a.view(np.uint32) != b.view(np.uint32)
        assert not bad.any(), (w, h, k, int(bad.sum()))
    assert g.stats()["jacobi_kernel"] == fluid_gb300.JACOBI_KERNEL_DATAFLOW
