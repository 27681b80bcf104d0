"""The azimuthal transforms at every length they are built for (16 to 512 samples), on grids
whose column counts leave a partial tile: forward (density and moments, warm-start potential)
and inverse (axis and equator conditions, effective potential) through solves against the
oracle, with the regular and the dense register budget."""
import numpy as np
import pytest

from tests.helpers import rel_l2, smooth_density

pytestmark = pytest.mark.gpu

POT_TOL = 1e-12  # the FP64 bar of every drop-in test
S_TOL = 1e-13    # the bar of the boundary moments


@pytest.mark.parametrize("dense", ["0", "1"])
@pytest.mark.parametrize("isym", [1, 2, 3])
@pytest.mark.parametrize("numphi", [16, 32, 64, 128, 256, 512])
def test_every_length(oracle_mod, bph, monkeypatch, numphi, isym, dense):
    monkeypatch.setenv("BPH_FFT_DENSE", dense)
    for numr, numz in ((9, 7), (21, 14)):  # 35 and 228 interior columns, 63 and 294 with the frame
        dr = 1.0 / (numr - 2)
        o = oracle_mod.Oracle(numr, numz, numphi, dr, isym, 3)
        g = bph.PotentialSolver(numr, numz, numphi, dr, isym, 3)
        rho = smooth_density(numr, numz, numphi, dr, isym, seed=numphi + isym)
        po = o.potential_solver(rho, 0)
        assert rel_l2(g.potential_solver(rho, 0), po) <= POT_TOL
        assert rel_l2(g.moments_S(), o.moments_S()) <= S_TOL
        g.set_potential(po)
        rho = np.asfortranarray(np.roll(rho, 1, axis=2))
        pot, phieff = g.potential_solver_phieff(rho, 2, 0.7)
        po = o.potential_solver(rho, 2)
        assert rel_l2(pot, po) <= POT_TOL
        rhf = (np.arange(1, numr + 1) - 1.5) * dr
        assert rel_l2(phieff, po - 0.5 * 0.7 ** 2 * rhf[:, None, None] ** 2) <= POT_TOL
        g.close()
        o.close()
