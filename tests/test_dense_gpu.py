"""The kernels with cusp replacement and three-body terms at four blocks per SM:
chosen when that saves whole waves of walkers (moves of spins up to 16) or the
walkers fill more than one wave (full evaluations), against the oracle just
above one wave of the others, where the last blocks are partly filled."""
import dataclasses

import numpy as np
import pytest

from qmcbeaver_b200.system import make_random_molecule, with_three_body
from test_rows64_gpu import _check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,W,cusp", [(2, 2001, True), (6, 2001, False), (17, 1999, True), (32, 2001, False)])
def test_evaluations_of_many_walkers_match_oracle(ne, W, cusp):
    s = with_three_body(make_random_molecule(ne, max(1, ne // 6), 3 * ne, 5.0 + ne / 12, (1, 6, 7, 8), seed=ne), seed=4)
    s = dataclasses.replace(s, replace_cusps=cusp)
    _check(s, W, [0, s.n_alpha - 1, ne - 1], np.array([0, 31, 1184, W - 1]))
