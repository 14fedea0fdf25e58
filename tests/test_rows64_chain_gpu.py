"""Chains whose proposals and orbital rows come from the batched FP64 rows
kernel (which proposes a walker's move a second time, for the rows): the walkers
of a handle large enough to use it follow the chain of a handle that is not, and
hold the energies of fresh evaluations."""
import dataclasses

import numpy as np
import pytest

from helpers import PARITY_RTOL, cond_bounds, slater_conditions
from qmcbeaver_b200.api import QMCB200Functions
from qmcbeaver_b200.desc import run_params
from qmcbeaver_b200.system import make_random_molecule, make_system, with_cambridge2, with_three_body

pytestmark = pytest.mark.gpu


def _fresh(s, w, n):
    g = QMCB200Functions(s, n, qf_modification=2, dt=0.01)
    out = g.evaluate(np.arange(n), w["R"][:n], -1)
    g.close()
    ok = out["status"] == 0
    # up to 25 updates since the last refresh: their rounding (1e-15 x condition
    # numbers below 1e6), relative to the Laplacian that E_L cancels from
    err = np.abs(w["e_local"][:n] - out["e_local"]) / np.maximum(np.abs(out["lap"]), 1.0)
    assert np.median(err[ok]) < 1e-12 and np.max(err[ok]) < 1e-8
    assert np.max(np.abs(w["log_abs_psi"][:n] - out["log_abs_psi"])[ok]) < 1e-8


@pytest.mark.parametrize("kind,sampling", [("34", 1), ("68", 0), ("34", 2), ("10", 2), ("10 three-body", 2),
                                           ("10 cusps", 1)])
def test_large_handles_follow_the_chain_of_small_ones(kind, sampling):
    ne = int(kind.split()[0])
    s = make_system("vmc_water_10e", seed=1) if ne == 10 else \
        make_random_molecule(ne, ne // 6, 3 * ne, 5.0 + ne / 12, (1, 6, 7, 8), seed=ne)
    if kind.endswith("three-body"):
        s = with_three_body(with_cambridge2(s, seed=2), seed=4)
    if kind.endswith("cusps"):
        s = dataclasses.replace(s, replace_cusps=True)
    W, few, steps = 3201, 9, 40
    R = s.initial_positions(W, seed=2, sigma=0.7)
    got = []
    for n in (W, few):
        f = QMCB200Functions(s, n, run_params(dt=0.01, seed=17, rel_cutoff=0.0, refresh_interval=25, sampling=sampling,
                                              qf_modification=2))
        f.set_profiling(True)
        f.init_walkers(R[:n])
        f.run_steps(3, steps)
        got.append(f.get_walkers())
        assert f.kernel_stats()["rows_prep"]["launches"] == (steps if n == W else 0)
        f.close()
    many, one = got
    # the same operations on the same random numbers: a kernel's own order of
    # the drift's few products may differ in the last bit
    assert np.max(np.abs(many["R"][:few] - one["R"])) < 1e-9
    assert np.max(np.abs(many["e_local"][:few] - one["e_local"]) / np.maximum(np.abs(one["e_local"]), 1.0)) < 1e-7
    if not kind.endswith("cusps"):
        _fresh(s, many, W)


def test_spins_above_64_take_the_rows_at_any_number_of_walkers():
    from oracle.evaluators import OracleEvaluator
    s = make_random_molecule(132, 20, 270, 16.0, (1, 6, 7, 8), seed=132)
    W, steps = 12, 72
    f = QMCB200Functions(s, W, run_params(dt=0.01, seed=17, rel_cutoff=0.0, refresh_interval=25, sampling=1,
                                          qf_modification=2))
    f.set_profiling(True)
    f.init_walkers(s.initial_positions(W, seed=2, sigma=0.7))
    f.run_steps(3, steps)  # the last step ends with a refresh: inverses of the rows that the moves stored
    assert f.kernel_stats()["rows_prep"]["launches"] == steps
    w = f.get_walkers()
    f.close()
    orc = OracleEvaluator(s, qf_mod=2, dt=0.01)
    ws = orc.new_walkers(W)
    orc.evaluate(ws, w["R"], -1)
    ref = orc.results(ws)
    slope, limit = cond_bounds(s)
    cond = slater_conditions(orc, ws, s)
    tol = np.where(cond >= limit, np.maximum(PARITY_RTOL, slope * cond), PARITY_RTOL)
    amp = (np.abs(ref["lap"]) / 2 + np.abs(ref["potential"])) / np.maximum(np.abs(ref["e_local"]), 1.0)
    err = np.abs(w["e_local"] - ref["e_local"]) / np.maximum(np.abs(ref["e_local"]), 1.0)
    assert np.all(err <= tol * np.maximum(amp, 1.0))
