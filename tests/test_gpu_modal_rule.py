"""Which form of the FP64 ADI a schedule takes (half-steps or the vertical eigenbasis), and that
short schedules and tall slots give the oracle's potential in either."""
import numpy as np
import pytest

from tests.helpers import rel_l2, smooth_density

pytestmark = pytest.mark.gpu

POT_TOL = 1e-12  # the FP64 bar of every drop-in test


def _grid(g):
    return (g[0], g[1], g[2], 1.0 / max(g[0] - 4, 2), g[3], g[4])


def _step_kernels(s, rho, nsteps):
    """Kernels of one explicit-count solve on device arrays."""
    import torch

    d = torch.from_numpy(np.ascontiguousarray(rho.ravel(order="F"))).cuda()
    pot = torch.empty_like(d)
    s.solve_nsteps_device(d, pot, nsteps, False)
    before = s.launch_count
    s.solve_nsteps_device(d, pot, nsteps, False)
    s.synchronize()
    return s.launch_count - before


# small slots (the eigenbasis from one step on, up to 64 radii and 48 heights), segmented, a thread per
# line, grid-wide panels, warp-cooperative; the first schedule length in the eigenbasis
GRIDS = [((18, 18, 16, 2, 6), 1), ((66, 50, 16, 2, 6), 1), ((66, 51, 16, 2, 6), 2), ((67, 45, 32, 3, 6), 2),
         ((90, 146, 16, 1, 5), 2), ((202, 152, 16, 2, 4), 2), ((66, 66, 16, 2, 4), 8)]


@pytest.mark.parametrize("grid,first", GRIDS, ids=["x".join(map(str, g[:3])) for g, _ in GRIDS])
def test_short_schedules(oracle_mod, bph, monkeypatch, grid, first):
    """A schedule of one step does not pay for transforms that cost more than it: it launches the
    half-step form's kernels.  One to three steps match the oracle's."""
    g = _grid(grid)
    rho = smooth_density(*g[:5], seed=3)
    with monkeypatch.context() as m:
        m.setenv("BPH_ADI_MODAL", "0")
        half = bph.PotentialSolver(*g)
        assert half.info()["adi_modal"] == 0
        kernels = _step_kernels(half, rho, 1)
        half.close()
    s = bph.PotentialSolver(*g)
    assert s.info()["adi_modal"] == first
    assert (_step_kernels(s, rho, 1) == kernels) == (first > 1)
    o = oracle_mod.Oracle(*g)
    assert rel_l2(s.potential_solver(rho, 0), o.potential_solver(rho, 0)) <= POT_TOL
    for n in (1, 2, 3):
        rho = np.asfortranarray(np.roll(rho, 1, axis=2))
        assert rel_l2(s.solve_nsteps(rho, n, False), o.solve_nsteps(rho, n, False)) <= POT_TOL
    s.close()
    o.close()


@pytest.mark.parametrize("tune", ["1", "0"], ids=["timed", "untimed"])
@pytest.mark.parametrize("grid", [(12, 300, 16, 1, 4), (8, 200, 32, 2, 6), (20, 146, 16, 3, 3), (30, 402, 16, 2, 4)],
                         ids=lambda g: "x".join(map(str, g[:3])))
def test_tall_slots(oracle_mod, bph, monkeypatch, grid, tune):
    """Tall slots take the form the set-up timed as the faster for the schedule (untimed: half-steps
    below eight); warm, cold and batched solves match the oracle."""
    monkeypatch.setenv("BPH_AUTOTUNE", tune)
    g = _grid(grid)
    s = bph.PotentialSolver(*g)
    o = oracle_mod.Oracle(*g)
    b = bph.Batch(s, capacity=2)
    first = s.info()["adi_modal"]
    assert first == 8 if tune == "0" else 2 <= first <= 64
    rho = smooth_density(*g[:5], seed=5)
    want = o.potential_solver(rho, 0)
    assert rel_l2(s.potential_solver(rho, 0), want) <= POT_TOL
    assert all(rel_l2(p, want) <= POT_TOL for p in b.solve([rho, rho], 0))
    rho = np.asfortranarray(np.roll(rho, 1, axis=2))
    want = o.potential_solver(rho, 2)
    assert rel_l2(s.potential_solver(rho, 2), want) <= POT_TOL
    assert all(rel_l2(p, want) <= POT_TOL for p in b.solve([rho, rho], 2))
    b.close()
    s.close()
    o.close()
