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


class _Filled:
    """All but `room` bytes of the device's free memory taken."""

    def __init__(self, room):
        import torch

        self.torch, self.held = torch, []
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        for unit in (1 << 30, 1 << 26, 1 << 22):
            free = torch.cuda.mem_get_info()[0]
            n = max(free - room, 0) // unit
            if n:
                self.held.append(torch.empty(n * unit, dtype=torch.uint8, device="cuda"))

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.torch.cuda.synchronize()
        self.held.clear()
        self.torch.cuda.empty_cache()


def _host(rho):
    import torch

    return torch.from_numpy(np.ascontiguousarray(rho.ravel(order="F"))).cuda()


MB = 1 << 20


def test_refused_converged_solve_leaves_the_state(bph, monkeypatch):
    """A cold mixed solve for whose FP32 work arrays there is no room is refused before it clears the
    potential that the next warm solve starts from."""
    g = (202, 152, 128, 1.0 / 198.0, 2, 4)  # work arrays: 61 MB a context, 4 x 31 MB for a batch of 2
    monkeypatch.setenv("BPH_ADI_MODAL", "0")
    rhos = [np.asfortranarray(smooth_density(*g[:5], seed=80 + i)) for i in range(2)]
    dev = [_host(r) for r in rhos]
    out = {}
    for refused in (False, True):
        s = bph.PotentialSolver(*g)
        b = bph.Batch(s, capacity=2)
        pot, pots = dev[0].clone(), [d.clone() for d in dev]
        s.potential_solver_device(dev[0], pot, 0)
        b.solve_device(dev, pots, 0)
        s.solve_nsteps_device(dev[0], pot, 10, False)  # the cycle's schedule, ahead
        if refused:
            with _Filled(24 * MB):
                with pytest.raises(bph.BphError) as err:
                    s.solve_converged_device(dev[1], pot, 10, True, 1e-9, 5, mixed=True)
                assert err.value.code == bph.BPH_ERR_NOMEM
                with pytest.raises(bph.BphError) as err:
                    b.solve_converged_device(dev[::-1], pots, 10, True, 1e-9, 5, mixed=True)
                assert err.value.code == bph.BPH_ERR_NOMEM
        s.potential_solver_device(dev[1], pot, 2)
        b.solve_device(dev[::-1], pots, 2)
        s.synchronize()
        out[refused] = [p.cpu().numpy() for p in [pot] + pots]
        b.close()
        s.close()
    for a, w in zip(out[True], out[False]):
        assert np.array_equal(a, w)


def test_mixed_batches_hold_no_fp64_array(bph):
    """Mixed converged solves in the vertical eigenbasis keep the modal potential (and, for slots
    without the grid-wide scratch, the residual); the FP64 form's earlier potential is allocated by
    the first FP64 solve.  Both forms work in either order."""
    for g, arrays in ((LARGE[0], 1), ((40, 30, 64, 1.0 / 36.0, 2, 16), 2)):
        rhos = [np.asfortranarray(smooth_density(*g[:5], seed=90 + i)) for i in range(3)]
        out = {}
        for first in ("mixed", "fp64"):
            s = bph.PotentialSolver(*g)
            s.set_mixed_adi(MIXED_ADI_GLOBAL)
            b = bph.Batch(s, capacity=3)
            b.solve(rhos, 0)  # the host arrays' staging
            before = b.device_bytes
            pots, sizes = {}, {}
            for form in ("mixed", "fp64") if first == "mixed" else ("fp64", "mixed"):
                pots[form], _ = b.solve_converged(rhos, 10, True, 1e-11, 60, mixed=form == "mixed")
                sizes[form] = b.device_bytes - before
            out[first] = pots
            slot_arrays = 3 * 8 * g[0] * g[1] * g[2]  # a modal array is smaller than a slot array
            if first == "mixed":
                assert sizes["mixed"] <= arrays * slot_arrays + MB
                assert sizes["fp64"] <= (arrays + 1) * slot_arrays + MB
            b.close()
            s.close()
        for form in ("mixed", "fp64"):
            for a, w in zip(out["mixed"][form], out["fp64"][form]):
                assert np.array_equal(a, w)
        for a, w in zip(out["mixed"]["mixed"], out["mixed"]["fp64"]):
            assert rel_l2(a, w) <= 1e-9  # tolerance 1e-11 of an update, each cycle reducing it


def test_optional_arrays_give_way(bph):
    """What a converged solve holds only to run in the vertical eigenbasis does not cost a later call
    its staging arrays: with room for these only in its place the host-array calls succeed, and the
    converged solve after them."""
    g = (101, 75, 128, 1.0 / 97.0, 2, 8)  # batch of 16: staging 248 MB, optional arrays 3 x 115 MB
    big = (250, 40, 512, 1.0 / 246.0, 2, 8)  # context: staging 2 x 41 MB, optional array 39 MB
    rho, many = smooth_density(*big[:5], seed=100), [smooth_density(*g[:5], seed=101 + i) for i in range(16)]
    out = {}
    for scarce in (False, True):
        s, one = bph.PotentialSolver(*g), bph.PotentialSolver(*big)
        b = bph.Batch(s, capacity=16)
        dev, pots = [_host(r) for r in many], [_host(r) for r in many]
        d, pot = _host(rho), _host(rho)
        b.solve_converged_device(dev, pots, 10, True, 1e-9, 60)
        one.solve_converged_device(d, pot, 10, True, 1e-9, 60)
        s.synchronize()
        one.synchronize()
        got = []
        if scarce:
            with _Filled(100 * MB):
                got += b.solve(many, 2)
                got += b.solve_converged(many, 10, False, 1e-11, 60)[0]
            with _Filled(60 * MB):
                got.append(one.potential_solver(rho, 2))
                got.append(one.solve_converged(rho, 10, False, 1e-11, 60)[0])
        else:
            got += b.solve(many, 2) + b.solve_converged(many, 10, False, 1e-11, 60)[0]
            got += [one.potential_solver(rho, 2), one.solve_converged(rho, 10, False, 1e-11, 60)[0]]
        got += b.solve_converged(many, 10, True, 1e-11, 60)[0]
        got.append(one.solve_converged(rho, 10, True, 1e-11, 60)[0])
        out[scarce] = got
        b.close()
        s.close()
        one.close()
    for a, w in zip(out[True], out[False]):
        assert rel_l2(a, w) <= 1e-12


def test_converged_host_call_whose_staging_takes_the_optional_array(bph):
    """The FP64 converged form's optional array gives way to the staging of the very call that would
    use it: the call runs the half-step cycles."""
    g = (250, 40, 512, 1.0 / 246.0, 2, 8)  # staging 2 x 41 MB, optional array 39 MB with d_prev's 41
    rho = smooth_density(*g[:5], seed=130)
    out = []
    for scarce in (False, True):
        s = bph.PotentialSolver(*g)
        d, pot = _host(rho), _host(rho)
        s.solve_converged_device(d, pot, 10, True, 1e-11, 60)
        s.synchronize()
        if scarce:
            with _Filled(60 * MB):
                got = s.solve_converged(rho, 10, True, 1e-11, 60)
        else:
            got = s.solve_converged(rho, 10, True, 1e-11, 60)
        out.append((got[0], s.solve_converged(rho, 10, True, 1e-11, 60)[0]))
        s.close()
    assert rel_l2(out[1][0], out[0][0]) <= 1e-12 and rel_l2(out[1][1], out[0][1]) <= 1e-12


@pytest.mark.parametrize("room", [40, 60, 90, 130, 200])
def test_every_form_without_room_for_the_next(oracle_mod, bph, room):
    """Batches, schedules and converged solves created with little room left run whichever form's
    arrays fit, and give the oracle's potential; refused calls name the reason."""
    g = (101, 75, 128, 1.0 / 97.0, 2, 8)  # a slot array 7.6 MB; twelve steps' factors 18 MB, modal ones 8 MB more
    o = oracle_mod.Oracle(*g)
    rho = smooth_density(*g[:5], seed=120)
    s = bph.PotentialSolver(*g)
    warm = bph.PotentialSolver(*g)  # every kernel and the staging, once
    warm.potential_solver(rho, 0)
    warm.solve_nsteps(rho, 12, False)
    warm.solve_converged(rho, 10, True, 1e-9, 60)
    wb = bph.Batch(warm, capacity=2)
    wb.solve([rho] * 2, 0)
    wb.solve_converged([rho] * 2, 10, True, 1e-9, 60)
    wb.close()
    warm.close()
    s.potential_solver(rho, 0)
    want = o.potential_solver(rho, 0)
    refused = 0
    with _Filled(room * MB):
        for call in ("steps", "converged", "batch"):
            try:
                if call == "steps":
                    assert rel_l2(s.solve_nsteps(rho, 12, True), o.solve_nsteps(rho, 12, True)) <= 1e-12
                elif call == "converged":
                    s.solve_converged(rho, 10, True, 1e-11, 60)
                else:
                    b = bph.Batch(s, capacity=2)
                    assert all(rel_l2(p, want) <= 1e-12 for p in b.solve([rho] * 2, 0))
                    b.solve_converged([rho] * 2, 10, True, 1e-11, 60)
                    b.close()
            except bph.BphError as err:
                assert err.code == bph.BPH_ERR_NOMEM
                refused += 1
    assert rel_l2(s.potential_solver(rho, 0), want) <= 1e-12
    assert refused < 3 or room < 60
    s.close()
    o.close()
