"""Converged solves whose cycles run in the vertical eigenbasis: the stopping rule goes by the
change of the potential itself, as in the half-step forms, so no solve goes on for a tolerance
below the potential's rounding."""
import numpy as np
import pytest

from bipoly_hydro_b200.solver import MIXED_ADI_GLOBAL
from tests.helpers import rel_l2, smooth_density

pytestmark = pytest.mark.gpu

# dense and split transforms, segments of 8 and 16 radii, one and several line groups, every symmetry
GRIDS = [(40, 30, 64, 2, 16), (67, 34, 32, 1, 6), (50, 19, 32, 3, 6), (35, 21, 64, 2, 12), (131, 74, 16, 2, 5)]
IDS = ["x".join(map(str, g[:3])) + f"-isym{g[3]}" for g in GRIDS]


@pytest.mark.parametrize("graph", ["1", "0"], ids=["device-loop", "host-loop"])
@pytest.mark.parametrize("grid", GRIDS, ids=IDS)
def test_update_ends_at_rounding(bph, monkeypatch, grid, graph):
    """Tolerance zero, 100 cycles allowed.  FP64: the loop ends once a cycle leaves the potential
    as it is.  Mixed: at its rounding, at most two cycles after the FP32 refinement on the same
    half-steps ends (which stagnates there; a cycle reduces the error several times)."""
    monkeypatch.setenv("BPH_CONV_GRAPH", graph)
    g = (grid[0], grid[1], grid[2], 1.0 / (grid[0] - 4), grid[3], grid[4])
    rhos = [np.asfortranarray(smooth_density(*g[:5], seed=40 + i)) for i in range(2)]
    cycles = {}
    for form in ("modal", "half"):
        if form == "half":
            monkeypatch.setenv("BPH_ADI_MODAL", "0")
        s = bph.PotentialSolver(*g)
        b = bph.Batch(s, capacity=2)
        ref, _ = s.solve_converged(rhos[0], 10, True, 1e-13, 60)
        if form == "modal":
            pot, one = s.solve_converged(rhos[0], 10, True, 0.0, 100)
            pots, many = b.solve_converged(rhos, 10, True, 0.0, 100)
            assert one.cycles < 100 and many.cycles < 100
            assert rel_l2(pot, ref) <= 1e-12 and rel_l2(pots[0], ref) <= 1e-12
        s.set_mixed_adi(MIXED_ADI_GLOBAL)
        pot, one = s.solve_converged_mixed(rhos[0], 10, True, 0.0, 100)
        pots, many = b.solve_converged(rhos, 10, True, 0.0, 100, mixed=True)
        assert rel_l2(pot, ref) <= 1e-12 and rel_l2(pots[0], ref) <= 1e-12
        cycles[form] = one.cycles, many.cycles
        b.close()
        s.close()
    assert cycles["modal"][0] <= cycles["half"][0] + 2 and cycles["modal"][1] <= cycles["half"][1] + 2


@pytest.mark.parametrize("grid", GRIDS, ids=IDS)
def test_mixed_cycles_are_the_refinement_iteration(bph, monkeypatch, grid):
    """The FP64 cycles that run in place of the grid-wide FP32 refinement take its half-steps, which
    end on a radial solve: no more cycles than it (one, where an update meets the tolerance by less
    than FP32 rounding), and less than a tenth of the residual at which half-steps that end on the
    vertical solve stagnate (its radially stiff components are the larger by that and more)."""
    g = (grid[0], grid[1], grid[2], 1.0 / (grid[0] - 4), grid[3], grid[4])
    rhos = [np.asfortranarray(smooth_density(*g[:5], seed=50 + i)) for i in range(2)]
    out = {}
    for form in ("modal", "half"):
        if form == "half":
            monkeypatch.setenv("BPH_ADI_MODAL", "0")
        s = bph.PotentialSolver(*g)
        s.set_mixed_adi(MIXED_ADI_GLOBAL)
        b = bph.Batch(s, capacity=2)
        _, cold = s.solve_converged_mixed(rhos[0], 10, True, 1e-11, 60)
        _, warm = s.solve_converged_mixed(rhos[1], 10, False, 1e-11, 60)
        _, many = b.solve_converged(rhos, 10, True, 1e-11, 60, mixed=True)
        out[form] = (cold, warm, many)
        if form == "half":
            _, vertical = s.solve_converged(rhos[0], 10, True, 1e-15, 30)
        b.close()
        s.close()
    for modal, half in zip(out["modal"], out["half"]):
        assert modal.residual <= 0.1 * vertical.residual
        assert modal.cycles <= half.cycles + 1


@pytest.mark.parametrize("kind", ["fp64", "global", "direct"])
def test_device_loop_ends_after_any_cycle(bph, monkeypatch, kind):
    """The device loop (a cycle, then passes of several) stops after 1 to 9 cycles like the host
    loop: the same count and the same potential, bit for bit."""
    g = (40, 30, 64, 1.0 / 36.0, 2, 16)
    rho = np.asfortranarray(smooth_density(*g[:5], seed=60))
    out = {}
    for graph in ("1", "0"):
        monkeypatch.setenv("BPH_CONV_GRAPH", graph)
        s = bph.PotentialSolver(*g)
        if kind != "fp64":
            s.set_mixed_adi(MIXED_ADI_GLOBAL if kind == "global" else 5)  # 5: the direct defect solve
        solve = s.solve_converged if kind == "fp64" else s.solve_converged_mixed
        out[graph] = [solve(rho, 10, True, 0.0, n) for n in range(1, 10)]
        s.close()
    for n, (a, b) in enumerate(zip(out["1"], out["0"]), 1):
        assert a[1].cycles == b[1].cycles and (a[1].cycles == n or kind != "fp64")
        assert np.array_equal(a[0], b[0])


@pytest.mark.parametrize("nsteps", [1, 2, 8, 15])
def test_cycle_lengths(bph, monkeypatch, nsteps):
    """Four cycles of any length are the half-steps' iterate: FP64 to rounding (1e-12, the drop-in's
    bar), the refinement's order to the FP32 cycles' rounding (2^-23 of an update, a few times over)
    where they reduce the error: cycles of one and two steps do not (they amplify FP32 rounding to
    1e-4 and 1e-6 of the potential, and the order's algebra is exact there as elsewhere)."""
    g = (50, 37, 32, 1.0 / 46.0, 2, 8)
    rhos = [np.asfortranarray(smooth_density(*g[:5], seed=150 + i)) for i in range(2)]
    out = {}
    for form in ("modal", "half"):
        if form == "half":
            monkeypatch.setenv("BPH_ADI_MODAL", "0")
        s = bph.PotentialSolver(*g)
        s.set_mixed_adi(MIXED_ADI_GLOBAL)
        b = bph.Batch(s, capacity=2)
        full = [s.solve_converged(rhos[0], nsteps, True, 0.0, 4)[0], s.solve_converged(rhos[1], nsteps, False, 0.0, 4)[0]]
        full += b.solve_converged(rhos, nsteps, True, 0.0, 4)[0]
        mixed = s.solve_converged_mixed(rhos[0], nsteps, True, 0.0, 4)
        out[form] = full, mixed
        b.close()
        s.close()
    for a, h in zip(out["modal"][0], out["half"][0]):
        assert rel_l2(a, h) <= 1e-12
    (a, ia), (h, ih) = out["modal"][1], out["half"][1]
    assert ia.cycles == ih.cycles
    assert nsteps <= 2 or rel_l2(a, h) <= 8 * 2.0 ** -23
