"""The FP64 ADI in the vertical eigenbasis (bph_modal.cu) against the oracle and
against the half-step kernels, at the edges of its tiles: radial lines around
one segment and one block, heights around the 8-row and 16-row fragments, odd
extents, every symmetry, and grids past its limits that keep the half-steps."""
import numpy as np
import pytest

from tests.helpers import rel_l2, smooth_density

pytestmark = pytest.mark.gpu

POT_TOL = 1e-12  # the FP64 bar of every drop-in test

GRIDS = [
    (5, 5, 16, 2, 3),      # 3 x 3 interior
    (10, 18, 16, 1, 4),    # one 8-radius segment, heights of one 16-row fragment
    (11, 19, 16, 2, 4),    # one radius and one height more
    (66, 35, 32, 3, 6),    # eight 8-radius segments, odd height
    (67, 34, 16, 2, 6),    # first 16-radius segments, one radius in the last
    (130, 27, 16, 1, 5),   # eight 16-radius segments
    (131, 98, 16, 2, 5),   # the production height beside a ninth segment
    (258, 20, 16, 2, 5),   # the longest line
    (259, 12, 16, 2, 5),   # past it: half-step kernels
    (20, 146, 16, 3, 3),   # heights past 128
    (20, 12, 16, 2, 4),    # split transforms: 21 = 3 x 7, second factor below one fragment
    (37, 24, 16, 3, 3),    # 45 = 5 x 9, factors not prime
    (34, 54, 32, 2, 6),    # 105 = 7 x 15 (and 3 x 35, 5 x 21)
    (21, 118, 16, 2, 4),   # 233: prime, dense
    (70, 194, 16, 2, 5),   # 385 = 7 x 55, the production height
]


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(map(str, g[:3])) + f"-isym{g[3]}")
def test_steps_match_oracle(oracle_mod, bph, grid):
    """Cold (20 steps), warm (5) and an explicit count, on one state."""
    numr, numz, numphi, isym, mmax = grid
    dr = 1.0 / max(numr - 4, 2)
    o = oracle_mod.Oracle(numr, numz, numphi, dr, isym, mmax)
    g = bph.PotentialSolver(numr, numz, numphi, dr, isym, mmax)
    rho = smooth_density(numr, numz, numphi, dr, isym, seed=7)
    assert rel_l2(g.potential_solver(rho, 0), o.potential_solver(rho, 0)) <= POT_TOL
    rho = np.asfortranarray(np.roll(rho, 1, axis=2) * 1.01)
    assert rel_l2(g.potential_solver(rho, 2), o.potential_solver(rho, 2)) <= POT_TOL
    assert rel_l2(g.solve_nsteps(rho, 9, False), o.solve_nsteps(rho, 9, False)) <= POT_TOL
    g.close()
    o.close()


@pytest.mark.parametrize("grid", [(35, 21, 64, 2, 12), (67, 34, 32, 1, 6), (50, 19, 32, 3, 6)],
                         ids=["isym2", "isym1", "isym3"])
def test_converged_and_batches_match_half_steps(bph, monkeypatch, grid):
    """Converged solves (cycle count and potential), warm batches with an instance map and a
    batch larger than one pass of the work array, against BPH_ADI_MODAL=0."""
    numr, numz, numphi, isym, mmax = grid
    dr = 1.0 / (numr - 4)
    rhos = [np.asfortranarray(smooth_density(numr, numz, numphi, dr, isym, seed=20 + i)) for i in range(5)]
    out = {}
    for form in ("modal", "half"):
        if form == "half":
            monkeypatch.setenv("BPH_ADI_MODAL", "0")
        g = bph.PotentialSolver(numr, numz, numphi, dr, isym, mmax)
        batch = bph.Batch(g, capacity=70)
        cold = batch.solve(rhos, 0)
        some = batch.solve_instances([4, 1], [rhos[0], rhos[2]], 2)
        many = batch.solve([rhos[i % 5] for i in range(70)], 0)
        conv, info = batch.solve_converged(rhos, 10, False, 1e-11, 60)
        single, one = g.solve_converged(rhos[0], 10, True, 1e-11, 60)
        again, two = g.solve_converged(rhos[1], 10, False, 1e-11, 60)
        out[form] = (cold + some + many + conv + [single, again], (info.cycles, one.cycles, two.cycles))
        batch.close()
        g.close()
    assert out["modal"][1] == out["half"][1]
    for a, b in zip(out["modal"][0], out["half"][0]):
        assert rel_l2(a, b) <= POT_TOL


def test_long_schedule_at_the_production_grid(oracle_mod, bph):
    """130x98x256 takes the modal form past seven steps: nine warm steps from a cold solve."""
    from bipoly_hydro_b200 import fields

    grid = (130, 98, 256, 1.0 / 126.0, 2, 30)
    rho = fields.bipolytrope_pair()
    o = oracle_mod.Oracle(*grid)
    g = bph.PotentialSolver(*grid)
    assert rel_l2(g.potential_solver(rho, 0), o.potential_solver(rho, 0)) <= POT_TOL
    rho = fields.rotate(rho)
    assert rel_l2(g.solve_nsteps(rho, 9, False), o.solve_nsteps(rho, 9, False)) <= POT_TOL
    g.close()
    o.close()
