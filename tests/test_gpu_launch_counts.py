"""Launch counts of a plan whose cold and warm solves run different forms of the ADI: each
replay adds its own kind's kernels to the context's count, and the plan reports those of
the kind launched last."""
import pytest

pytestmark = pytest.mark.gpu


def test_plan_counts_per_kind(bph):
    import torch

    grid = (66, 66, 16, 1.0 / 62.0, 2, 4)  # 5 steps in half-step form, 20 in the vertical eigenbasis
    solver = bph.PotentialSolver(*grid)
    solver.set_stream(torch.cuda.current_stream())
    batch = bph.Batch(solver, capacity=2)
    rho = [torch.rand(66 * 66 * 16, dtype=torch.float64, device="cuda") for _ in range(2)]
    pot = [torch.empty_like(r) for r in rho]
    want = {}
    for tstep in (0, 2):  # the kernels of one batched call
        batch.solve_device(rho, pot, tstep)
        before = solver.launch_count
        batch.solve_device(rho, pot, tstep)
        want[tstep] = solver.launch_count - before
    assert want[0] != want[2]
    plan = bph.Plan([(batch, rho, pot)])
    assert plan.launches == 0
    for tstep in (0, 2, 0, 2, 2, 0):
        before = solver.launch_count
        plan.launch(tstep, torch.cuda.current_stream())
        assert solver.launch_count - before == want[tstep]
        assert plan.launches == want[tstep]
    plan.synchronize(torch.cuda.current_stream())
    plan.close()
    solver.close()
