"""The FP64 half-step kernels and the grid-wide FP32 refinement, which grids past the vertical
eigenbasis's limits and schedules below its threshold run: whole schedules of each kernel against
the oracle with the eigenbasis off (BPH_ADI_MODAL=0), and past its limit of 256 radii without it;
single, batched, planned and served."""
import numpy as np
import pytest

from bipoly_hydro_b200.solver import MIXED_ADI_FORWARD, MIXED_ADI_GLOBAL
from tests.helpers import rel_l2, smooth_density

pytestmark = pytest.mark.gpu

POT_TOL = 1e-12  # the FP64 bar of every drop-in test
WARP, SEGMENTED, ONCHIP, GRID_WIDE = 1, 2, 3, 4

KERNELS = [
    ((66, 66, 64, 1.0 / 62.0, 2, 30), WARP),
    ((34, 26, 64, 1.0 / 30.0, 2, 30), SEGMENTED),
    ((90, 146, 16, 1.0 / 86.0, 1, 5), ONCHIP),
    ((202, 152, 16, 1.0 / 198.0, 2, 4), GRID_WIDE),
    ((261, 14, 16, 1.0 / 257.0, 3, 3), SEGMENTED),  # more than 256 radii: no eigenbasis to turn off
    ((301, 132, 16, 1.0 / 297.0, 2, 4), GRID_WIDE),
]
IDS = ["x".join(map(str, g[:3])) for g, _ in KERNELS]
LARGE = [KERNELS[3][0], KERNELS[5][0]]


def _half(bph, monkeypatch, grid, kernel):
    if grid[0] - 2 <= 256:
        monkeypatch.setenv("BPH_ADI_MODAL", "0")
    s = bph.PotentialSolver(*grid)
    info = s.info()
    assert info["adi_modal"] == 0 and info["adi_kernel"] == kernel
    return s


def _rho(grid, seed):
    return np.asfortranarray(smooth_density(*grid[:5], seed=seed))


@pytest.mark.parametrize("grid,kernel", KERNELS, ids=IDS)
def test_schedules_match_oracle(oracle_mod, bph, monkeypatch, grid, kernel):
    """Cold (20 steps), warm (5) and explicit counts."""
    s, o = _half(bph, monkeypatch, grid, kernel), oracle_mod.Oracle(*grid)
    rho = _rho(grid, 7)
    assert rel_l2(s.potential_solver(rho, 0), o.potential_solver(rho, 0)) <= POT_TOL
    rho = np.asfortranarray(np.roll(rho, 1, axis=2) * 1.01)
    assert rel_l2(s.potential_solver(rho, 2), o.potential_solver(rho, 2)) <= POT_TOL
    for n in (1, 9):
        assert rel_l2(s.solve_nsteps(rho, n, False), o.solve_nsteps(rho, n, False)) <= POT_TOL
    s.close()
    o.close()


@pytest.mark.parametrize("prefetch", ["0", "1"])
def test_segmented_factor_prefetch(oracle_mod, bph, monkeypatch, prefetch):
    """The segmented kernel over whole schedules with and without bulk-copy factor prefetch."""
    monkeypatch.setenv("BPH_ADI_PREFETCH", prefetch)
    grid = KERNELS[1][0]
    s, o = _half(bph, monkeypatch, grid, SEGMENTED), oracle_mod.Oracle(*grid)
    assert s.info()["adi_prefetch"] == (3 if prefetch == "1" else 0)
    rho = _rho(grid, 8)
    assert rel_l2(s.potential_solver(rho, 0), o.potential_solver(rho, 0)) <= POT_TOL
    rho = np.asfortranarray(np.roll(rho, 1, axis=2))
    assert rel_l2(s.potential_solver(rho, 2), o.potential_solver(rho, 2)) <= POT_TOL
    s.set_mixed_adi(MIXED_ADI_FORWARD)
    full, _ = s.solve_converged(rho, 10, True, 1e-13, 100)
    assert rel_l2(s.solve_converged_mixed(rho, 10, True, 1e-13, 100)[0], full) <= 1e-9
    s.close()
    o.close()


@pytest.mark.parametrize("grid,kernel", KERNELS, ids=IDS)
def test_converged_and_refined(oracle_mod, bph, monkeypatch, grid, kernel):
    """FP64 converged against the oracle's, and the FP32 refinement in global memory against FP64
    (1e-9, the bar of the mixed form), cold and warm."""
    s, o = _half(bph, monkeypatch, grid, kernel), oracle_mod.Oracle(*grid)
    s.set_mixed_adi(MIXED_ADI_GLOBAL)
    rho = _rho(grid, 9)
    want, _, _ = o.solve_converged(rho, 10, True, 1e-12, 60)
    full, _ = s.solve_converged(rho, 10, True, 1e-12, 60)
    assert rel_l2(full, want) <= 1e-9  # two iterations, each within a tolerance of 1e-12 an update
    assert rel_l2(s.solve_converged_mixed(rho, 10, True, 1e-12, 60)[0], full) <= 1e-9
    rho = np.asfortranarray(np.roll(rho, 1, axis=2))
    full, _ = s.solve_converged(rho, 10, False, 1e-12, 60)
    assert rel_l2(s.solve_converged_mixed(rho, 10, False, 1e-12, 60)[0], full) <= 1e-9
    s.close()
    o.close()


@pytest.mark.parametrize("grid", LARGE, ids=["202x152x16", "301x132x16"])
def test_grid_wide_batches_plans_and_servers(bph, monkeypatch, grid):
    """Every instance equals its own single solves: batched drop-in (an instance map too), batched
    converged FP64 and refined, a plan, and a server in mixed converged mode."""
    import torch

    n = 3
    rhos = [_rho(grid, 20 + i) for i in range(n)]
    moved = [np.asfortranarray(np.roll(r, 1, axis=2)) for r in rhos]
    s = _half(bph, monkeypatch, grid, GRID_WIDE)
    assert s.info()["mixed_kind"] == MIXED_ADI_GLOBAL
    one = [_half(bph, monkeypatch, grid, GRID_WIDE) for _ in range(n)]
    b = bph.Batch(s, capacity=n)
    for tstep, dens in ((0, rhos), (2, moved)):
        for i, p in enumerate(b.solve(dens, tstep)):
            assert rel_l2(p, one[i].potential_solver(dens[i], tstep)) <= POT_TOL
    got = b.solve_instances([2, 0], [rhos[2], rhos[0]], 3)
    assert rel_l2(got[0], one[2].potential_solver(rhos[2], 3)) <= POT_TOL
    assert rel_l2(got[1], one[0].potential_solver(rhos[0], 3)) <= POT_TOL
    full = [one[i].solve_converged(rhos[i], 10, True, 1e-12, 60)[0] for i in range(n)]
    for mixed in (False, True):
        pots, _ = b.solve_converged(rhos, 10, True, 1e-12, 60, mixed=mixed)
        assert all(rel_l2(p, f) <= 1e-9 for p, f in zip(pots, full))
    dev = [torch.from_numpy(np.ascontiguousarray(r.ravel(order="F"))).cuda() for r in rhos]
    out = [torch.empty_like(d) for d in dev]
    torch.cuda.synchronize()
    plan = bph.Plan([(b, dev, out)])
    stream = torch.cuda.Stream()
    for tstep in (0, 2):
        plan.launch(tstep, stream)
        plan.synchronize(stream)
        for i in range(n):
            p = out[i].cpu().numpy().reshape(rhos[i].shape, order="F")
            assert rel_l2(p, one[i].potential_solver(rhos[i], tstep)) <= POT_TOL
    plan.close()
    b.close()
    server = bph.Server(s, max_clients=2)
    server.set_converged(nsteps=10, tol=1e-12, max_cycles=60, mixed=True)
    clients = [server.open_client() for _ in range(2)]
    for i in (1, 0):
        pot, _ = server.wait(server.submit(clients[i], rhos[i]), timeout=120.0)
        assert rel_l2(pot, full[i]) <= 1e-9
    server.close()
    for x in one + [s]:
        x.close()
