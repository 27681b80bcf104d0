"""Device memory of the vertical-eigenbasis form: what it may add, and that every call still
succeeds where only the half-steps' arrays fit."""
import numpy as np
import pytest

from bipoly_hydro_b200.solver import MIXED_ADI_GLOBAL
from tests.helpers import rel_l2, smooth_density

pytestmark = pytest.mark.gpu

# slots beyond shared memory: odd and even heights (the modal array pads the odd ones)
LARGE = [(202, 152, 32, 1.0 / 198.0, 2, 4), (201, 153, 32, 1.0 / 198.0, 1, 4)]


def _modal_bytes(g):
    numr, numz, numphi = g[:3]
    return 8 * numphi * (numr - 2) * ((numz - 1) // 2 * 2)


@pytest.mark.parametrize("g", LARGE, ids=["even", "odd"])
def test_large_slots_keep_no_array_beside_their_scratch(bph, monkeypatch, g):
    """The scratch of the grid-wide half-steps holds the modal arrays too: a context adds tables and
    factors only, a batch nothing, and its results do not change with what was in the scratch."""
    rhos = [np.asfortranarray(smooth_density(*g[:5], seed=70 + i)) for i in range(3)]
    used, out = {}, {}
    for form in ("modal", "half"):
        if form == "half":
            monkeypatch.setenv("BPH_ADI_MODAL", "0")
        s = bph.PotentialSolver(*g)
        assert s.info()["adi_kernel"] == 4  # grid-wide
        bytes0 = s.device_bytes
        b = bph.Batch(s, capacity=3)
        used[form] = bytes0, b.device_bytes
        s.solve_nsteps(rhos[0], 1, True)  # the scratch in use as such
        single = [s.potential_solver(rhos[0], 0), s.potential_solver(rhos[1], 2),
                  s.solve_converged(rhos[2], 10, False, 1e-11, 60)[0]]
        many = b.solve(rhos, 0) + b.solve_instances([2, 0], rhos[1:], 2)
        many += b.solve_converged(rhos, 10, False, 1e-11, 60)[0] + b.solve(rhos, 2)
        out[form] = single + many
        b.close()
        s.close()
    # factors: five words a radius, padded to 256 radii, for 5 and 20 steps and a cycle of 10
    factors = 8 * 35 * g[2] * 5 * 256
    assert used["modal"][0] - used["half"][0] <= factors + (1 << 20)
    assert used["modal"][1] == used["half"][1]
    for a, h in zip(out["modal"], out["half"]):
        assert rel_l2(a, h) <= 1e-12
