"""The vertical eigenbasis's split transforms by the factor that each height takes, asserted, so
that a change of the rule cannot drop one unseen: every first factor, second factors below one
fragment, not prime, and of several fragments, and heights whose factors the rule leaves."""
import numpy as np
import pytest

from tests.helpers import rel_l2, smooth_density

pytestmark = pytest.mark.gpu

POT_TOL = 1e-12  # the FP64 bar of every drop-in test

#: numz -> first factor of 2 (numz - 2) + 1 (0: dense)
HEIGHTS = {
    12: 0,   # 21 = 3 x 7: three products for the dense form's two
    21: 3,   # 39 = 3 x 13, the second factor below one fragment
    24: 0,   # 45 = 5 x 9: five products for six
    34: 5,   # 65 = 5 x 13
    45: 3,   # 87 = 3 x 29
    54: 7,   # 105 = 7 x 15, not prime (and 3 x 35, 5 x 21)
    66: 3,   # 129 = 3 x 43, two row tiles
    69: 5,   # 135 = 5 x 27 (3 x 45 has a common factor)
    98: 0,   # 193, prime
    122: 0,  # 241, prime
    194: 7,  # 385 = 7 x 55
}


@pytest.mark.parametrize("isym", [2, 3])
@pytest.mark.parametrize("numz", sorted(HEIGHTS))
def test_split_factor(oracle_mod, bph, numz, isym):
    g = (37, numz, 16, 1.0 / 33.0, isym, 3)
    s, o = bph.PotentialSolver(*g), oracle_mod.Oracle(*g)
    assert s.info()["modal_split"] == HEIGHTS[numz]
    rho = smooth_density(*g[:5], seed=numz)
    assert rel_l2(s.potential_solver(rho, 0), o.potential_solver(rho, 0)) <= POT_TOL
    rho = np.asfortranarray(np.roll(rho, 1, axis=2))
    assert rel_l2(s.solve_nsteps(rho, 9, False), o.solve_nsteps(rho, 9, False)) <= POT_TOL
    s.close()
    o.close()


def test_no_split_of_a_dirichlet_bottom(bph):
    """Without a reflecting bottom the transform is another one and stays dense."""
    s = bph.PotentialSolver(37, 54, 16, 1.0 / 33.0, 1, 3)
    assert s.info()["modal_split"] == 0
    s.close()
