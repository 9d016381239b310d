"""V_KS on grids whose edges take every line transform of the density grid:
each compile-time plan on some axis, and an edge without one (8) first, in the
middle and last, where the real input and output steps run on their own.

Against the numpy restatement; rho(G) 1e-13, V_KS and energies 1e-12 as on the
other density grids (FP64 transforms of at most 128 points an axis)."""
import numpy as np
import pytest

from conftest import rel_l2
from oracle import vks as V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xc", [1, 0])
@pytest.mark.parametrize("grid,ecut", [((16, 18, 27), 9.0), ((36, 12, 24), 4.0), ((8, 48, 64), 2.0), ((54, 8, 81), 2.0),
                                       ((72, 96, 8), 2.0), ((108, 32, 128), 9.0)])
def test_vks_edges(pkg, wl, grid, ecut, xc):
    s = wl.make_system(1, grid, disp_sigma=0.05, seed=4, with_kb=False)
    ka, kb, kc, _, _ = pkg.setkvec3d_sm(s["hmat"], ecut, list(grid))
    vtab, gmin, dg, gz = wl.local_table()
    g = pkg.DensityGrid(*grid, s["hmat"], ka, kb, kc)
    g.set_local(s["pos"], vtab, gmin, dg, gz)
    vre, vim = V.vext(s["hmat"], ka, kb, kc, s["pos"], vtab, vtab.shape[1], gmin, dg, gz)
    rho = 0.5 + np.random.default_rng(2).random(int(np.prod(grid)))
    rho *= s["num_elec"] / rho.mean()
    for _ in range(2):  # the second call finds the work grid as the first left it
        v, rre, rim, e = g.vks_from_rho(rho, pkg.SDFT_XC_PZ_LDA if xc else 0)
        ov, orr, ori, oe = V.vks_from_rho(grid, s["hmat"], ka, kb, kc, vre, vim, rho, xc=bool(xc))
        assert rel_l2(rre, orr) < 1e-13 and rel_l2(rim, ori) < 1e-13
        assert rel_l2(v, ov) < 1e-12
        assert np.all(np.abs(e - oe) <= 1e-12 * np.abs(oe) + (0.0 if xc else 1e-300))
    g.close()
