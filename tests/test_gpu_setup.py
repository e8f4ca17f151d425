"""The piecewise setup of the pressure system (k_setup_pieces, grids of 2^20
cells and more) against the oracle: sides
with every remainder of 4 columns, holes in the mask, no sweeps and some."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,iters", [(1022, 1022, 0), (1024, 1023, 8), (1040, 1024, 3), (1031, 1025, 9)])
def test_large_setup_bitwise(w, h, iters):
    import fluid_gb300
    from oracle.pyoracle import OracleFluid

    p = dict(scheme=1, num_iters=iters, early_exit=False)
    g = fluid_gb300.Fluid(1.0, w, h, 1.0, **p)
    o = OracleFluid(1.0, w, h, 1.0, prec=32, threads=8, **p)
    S = (np.random.default_rng(w).random(g.numCells) > 0.01).astype(np.float32)
    for f in (g, o):
        f.S[:] = S
        scenes.random_state(f, seed=iters + 1, amp=1.0)
        f.makeIncompressible(iters, 0.1)
    for k in ("U", "V", "p"):
        a, b = getattr(g, k), getattr(o, k)
        bad = a.view(np.uint32) != b.view(np.uint32)
        assert not bad.any(), (w, h, k, int(bad.sum()))
