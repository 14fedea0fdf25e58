"""Calls with more walkers than 65,535 tiles of 32 hold (the largest second or
third dimension of a launch grid): every walker is evaluated."""
import numpy as np
import pytest

from qmcbeaver_b200.api import QMCB200Functions
from qmcbeaver_b200.system import make_random_molecule

pytestmark = pytest.mark.gpu


def test_two_million_walkers():
    s = make_random_molecule(2, 1, 5, 4.0, (2,), seed=2)
    W, few = 32 * 65535 + 40, 1024
    rng = np.random.default_rng(3)
    R0 = s.initial_positions(few, seed=1)
    pick = rng.integers(0, few, W)
    f, g = QMCB200Functions(s, W, qf_modification=2, dt=0.01), QMCB200Functions(s, few, qf_modification=2, dt=0.01)
    want = g.evaluate(np.arange(few), R0, -1)
    for R, w in ((R0, want), (R0 + 0.1, g.evaluate(np.arange(few), R0 + 0.1, -1))):
        got = f.evaluate(np.arange(W), R[pick], -1)
        for k in ("e_local", "log_abs_psi", "sign", "lap", "grad", "status"):
            assert np.array_equal(got[k], w[k][pick]), k
    f.init_walkers(R0[pick])
    assert np.array_equal(f.get_walkers()["e_local"], want["e_local"][pick])
    f.close()
    g.close()
