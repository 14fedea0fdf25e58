"""Inverses of the Slater matrices in register tiles: full evaluations against
the oracle at the sizes where the tiles change, a
matrix without pivots, and the refresh of a chain."""
import numpy as np
import pytest

from helpers import PARITY_RTOL, compare, cond_bounds, slater_conditions
from qmcbeaver_b200.api import QMCB200Functions
from qmcbeaver_b200.desc import run_params
from qmcbeaver_b200.system import make_random_molecule, make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 8, 9, 16, 17, 24, 25, 32, 33, 40, 41, 56, 57, 80, 81, 112, 113, 128])
def test_tiles_match_oracle(n):
    from oracle.evaluators import OracleEvaluator
    ne, W = 2 * n - 1, 5  # the other spin one smaller
    s = make_random_molecule(ne, max(1, ne // 8), 2 * n + 3, 5.0 + ne / 12, (1, 6, 7, 8), seed=n, orbitals="random")
    f = QMCB200Functions(s, W, qf_modification=2, dt=0.01)
    orc = OracleEvaluator(s, qf_mod=2, dt=0.01)
    R = s.initial_positions(W, seed=2, sigma=0.7)
    watched = [0, W - 1]
    ws = orc.new_walkers(len(watched))
    out = {k: v[watched] for k, v in f.evaluate(np.arange(W), R, -1).items()}
    orc.evaluate(ws, R[watched], -1)
    ref = orc.results(ws)
    cond = slater_conditions(orc, ws, s)
    slope, limit = cond_bounds(s)
    amp = (np.abs(ref["lap"]) / 2 + np.abs(ref["potential"])) / np.maximum(np.abs(ref["e_local"]), 1.0)
    for i in range(len(watched)):
        compare(out, ref, max(PARITY_RTOL, slope * cond[i]) if cond[i] >= limit else PARITY_RTOL,
                f"{n} electrons a spin, walker {watched[i]} (cond {cond[i]:.1e})",
                mask=np.arange(len(watched)) == i, kappa=amp)
    f.close()


def test_singular_matrix_is_flagged_alone():
    s = make_system("vmc_water_10e", seed=1)
    f = QMCB200Functions(s, 3, qf_modification=2, dt=0.01)
    R = s.initial_positions(3, seed=1)
    good = f.evaluate(np.arange(3), R, -1)
    R2 = R.copy()
    R2[1] += 1e3  # every basis function underflows: zero Slater matrices
    out = f.evaluate(np.arange(3), R2, -1)
    assert out["status"][1] & 1 and not out["status"][0] and not out["status"][2]
    for k in ("log_abs_psi", "sign", "e_local", "lap", "grad"):
        assert np.array_equal(out[k][[0, 2]], good[k][[0, 2]])
    f.close()


def test_refresh_keeps_the_chain():
    """A refreshed chain's energies equal fresh evaluations at its positions."""
    s = make_random_molecule(38, 6, 150, 8.0, (1, 6, 7, 8), seed=5)
    W = 24
    f = QMCB200Functions(s, W, run_params(sampling=1, qf_modification=2, dt=0.01, seed=3, refresh_interval=10,
                                          rel_cutoff=0.0))
    f.init_walkers(s.initial_positions(W, seed=2))
    f.run_steps(0, 50)
    w = f.get_walkers()
    g = QMCB200Functions(s, W, qf_modification=2, dt=0.01)
    out = g.evaluate(np.arange(W), w["R"], -1)
    # the refresh inverts rows carried over up to 50 moves unchanged: the same
    # matrices, equal up to their rounding (1e-15 x condition numbers < 1e6)
    assert np.max(np.abs(w["e_local"] - out["e_local"]) / np.maximum(np.abs(out["lap"]), 1.0)) < 1e-9
    assert np.max(np.abs(w["log_abs_psi"] - out["log_abs_psi"])) < 1e-8
    f.close()
    g.close()
