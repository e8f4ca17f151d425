"""The MULTIGRID scheme's levels where they can go wrong: odd sides whose last
child has no pair, coarsest levels of one warp's cells, of up to 1024 and of
more (thin grids), levels on either side of the bottom kernel's shared memory,
widths with every remainder of 4, random masks (coarse cells of one to four
children)."""
import numpy as np
import pytest

import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,iters,holes", [
    (16, 16, 2, 0.0), (17, 31, 2, 0.1), (10, 2000, 2, 0.04), (300, 10, 1, 0.0), (11, 5003, 2, 0.02),
    (93, 90, 3, 0.04), (188, 139, 2, 0.3), (240, 239, 1, 0.0), (265, 359, 3, 0.04),
    (1121, 961, 2, 0.1),
])
def test_multigrid_levels_bitwise(w, h, iters, holes):
    import fluid_gb300
    from oracle.pyoracle import OracleFluid

    p = dict(scheme=3, num_iters=iters, early_exit=False)
    g = fluid_gb300.Fluid(1.0, w, h, 1.0, **p)
    o = OracleFluid(1.0, w, h, 1.0, prec=32, threads=8, **p)
    S = (np.random.default_rng(w * h).random(g.numCells) >= holes).astype(np.float32)
    for f in (g, o):
        f.S[:] = S
        scenes.random_state(f, seed=iters, amp=1.0)
    for _ in range(2):
        for f in (g, o):
            f.makeIncompressible(iters, 0.1)
    for k in ("U", "V", "p"):
        a, b = getattr(g, k), getattr(o, k)
        bad = a.view(np.uint32) != b.view(np.uint32)
        assert not bad.any(), (w, h, k, int(bad.sum()))
    assert g.stats()["sweeps"] == iters
