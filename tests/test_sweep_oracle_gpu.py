"""Metropolis moves of the sweep kernel step by step against the oracle: the
step's records give every proposal, the oracle psi and the drifts at both ends,
and so the acceptance probability; the walkers after the step hold the oracle's
local energies."""
import numpy as np
import pytest

from helpers import PARITY_RTOL, cond_bounds, slater_conditions
from qmcbeaver_b200.api import QMCB200Functions
from qmcbeaver_b200.desc import run_params
from qmcbeaver_b200.system import make_random_molecule, make_system

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne,sampling,qf,dt", [(0, 0, 0, 0.09), (0, 1, 2, 0.01), (3, 1, 1, 0.02), (17, 1, 2, 0.01),
                                               (32, 1, 0, 0.01)])
def test_moves_match_oracle(ne, sampling, qf, dt):
    from oracle.evaluators import OracleEvaluator
    s = make_random_molecule(ne, max(1, ne // 5), 4 * ne + 1, 4.0 + ne / 10, (1, 6, 7, 8), seed=ne) if ne else \
        make_system("vmc_water_10e", seed=1)
    W, N, a = 21, s.n_electrons, 0.5
    f = QMCB200Functions(s, W, run_params(sampling=sampling, qf_modification=qf, qf_equal_a=a, dt=dt, seed=9,
                                          rel_cutoff=0.0))
    f.init_walkers(s.initial_positions(W, seed=3, sigma=0.7))
    f.set_profiling(True)
    orc = OracleEvaluator(s, qf_mod=qf, qf_a=a, dt=dt)
    ws, wt = orc.new_walkers(W), orc.new_walkers(W)
    slope, limit = cond_bounds(s)
    worst = np.zeros(W)
    accepted = checked = 0
    for step in range(1, N + 3):
        e = step % N
        R0 = f.get_walkers()["R"]
        rec, _ = f.run_step_configs(step)
        after = f.get_walkers()
        trial, old = rec[0::2], rec[1::2]
        Rt = trial[:, :3 * N].reshape(W, N, 3)
        assert np.array_equal(old[:, :3 * N].reshape(W, N, 3), R0)
        others = np.arange(N) != e
        assert np.array_equal(Rt[:, others], R0[:, others])
        orc.evaluate(ws, R0, -1)
        orc.evaluate(wt, Rt, -1)
        r0, rt = orc.results(ws), orc.results(wt)
        worst = np.maximum(worst, np.maximum(slater_conditions(orc, ws, s), slater_conditions(orc, wt, s)))
        ok = (worst < limit) & (r0["singular"] == 0) & (rt["singular"] == 0)
        log_p = 2 * (rt["log_abs_psi"] - r0["log_abs_psi"])
        if sampling == 1:
            # ln G(R' -> R) - ln G(R -> R'), the unmoved electrons' drifts among them
            fwd, rev = -dt * r0["mod_grad"], -dt * rt["mod_grad"]
            fwd[:, e] += Rt[:, e] - R0[:, e]
            rev[:, e] += R0[:, e] - Rt[:, e]
            log_p += (np.sum(fwd ** 2, (1, 2)) - np.sum(rev ** 2, (1, 2))) / (2 * dt)
        p = np.exp(np.minimum(log_p, 0.0))
        # 1e-10 of log|psi| and of the drifts, these 1 / (2 dt) times their squares
        assert np.max(np.abs(trial[ok, -1] - p[ok])) < 1e-8
        moved = np.array([not np.array_equal(after["R"][w], R0[w]) for w in range(W)])
        assert np.array_equal(after["R"], np.where(moved[:, None, None], Rt, R0))
        ref = {k: np.where(moved, rt[k], r0[k]) for k in ("e_local", "log_abs_psi", "lap", "potential")}
        amp = (np.abs(ref["lap"]) / 2 + np.abs(ref["potential"])) / np.maximum(np.abs(ref["e_local"]), 1.0)
        tol = np.maximum(PARITY_RTOL, slope * worst)
        assert np.all((np.abs(after["e_local"] - ref["e_local"]) / np.maximum(np.abs(ref["e_local"]), 1.0)
                       <= tol * np.maximum(amp, 1.0))[ok])
        assert np.all((np.abs(after["log_abs_psi"] - ref["log_abs_psi"]) <= tol)[ok])
        accepted += moved.sum()
        checked += ok.sum()
    assert checked > 0.5 * W * (N + 2) and 0 < accepted < W * (N + 2)
    k = f.kernel_stats()
    assert k["move"]["launches"] == N + 2 and k["rows_prep"]["launches"] == 0
    f.close()
