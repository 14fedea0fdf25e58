"""The sweep kernel (spins of up to 16 electrons, 16 walkers per CTA, all steps
between two branchings or refreshes in one launch) against the one-warp-per-
walker move kernel, which runs the same chain when the handle is made to keep
its inverses in device memory: every sampling, drift, reweighting and
correlation form it takes, at the edges of its tiles."""
import dataclasses

import numpy as np
import pytest

from qmcbeaver_b200.api import QMCB200Functions
from qmcbeaver_b200.desc import QMCB_DMC, QMCB_ECUT_BDJM_PUSH88, QMCB_ECUT_UMRIGAR93, run_params
from qmcbeaver_b200.system import make_random_molecule, make_system, with_cambridge2

pytestmark = pytest.mark.gpu


def _molecule(ne, jastrow=True):
    return make_random_molecule(ne, max(1, ne // 5), 4 * ne + 1, 4.0 + ne / 10, (1, 6, 7, 8), seed=ne, jastrow=jastrow)


def _compare(monkeypatch, s, W, steps, first=0, **kw):
    """`steps` steps by either kernel, the second's one by one: the same walkers.
    The two kernels add in different orders; a step's rounding (1e-15 times
    condition numbers below 1e6) grows to less than 1e-7 of the positions and,
    relative to the local energies, over the sweeps run here."""
    p = dict(dt=0.01, seed=11, rel_cutoff=0.0)
    p.update(kw)
    a = QMCB200Functions(s, 2 * W, run_params(**p))
    monkeypatch.setenv("QMCB_STAGED_INVERSE_MAX", "0")  # read when a handle is made
    b = QMCB200Functions(s, 2 * W, run_params(**p))
    R = s.initial_positions(W, seed=2)
    for f in (a, b):
        f.init_walkers(R)
    st = a.run_steps(first, steps)
    sums = np.zeros(5)
    for k in range(steps):
        one = b.run_steps(first + k, 1)
        sums += [one.sum_weight, one.sum_weight_energy, one.sum_accept, one.n_moves, one.n_singular]
    x, y = a.get_walkers(), b.get_walkers()
    assert len(x["weight"]) == len(y["weight"]) == st.n_walkers
    assert np.max(np.abs(x["R"] - y["R"])) < 1e-7
    for k in ("weight", "e_local", "log_abs_psi"):
        assert np.max(np.abs(x[k] - y[k]) / np.maximum(np.abs(y[k]), 1.0)) < 1e-6, k
    assert np.array_equal(x["sign"], y["sign"])
    assert st.n_moves == sums[3] and st.n_singular == sums[4]
    assert abs(st.sum_accept - sums[2]) < 1e-6 * max(1.0, sums[2])
    assert abs(st.sum_weight - sums[0]) < 1e-6 * max(1.0, sums[0])
    assert abs(st.sum_weight_energy - sums[1]) < 1e-5 * max(1.0, abs(sums[1]))
    for f in (a, b):
        f.close()


@pytest.mark.parametrize("ne,W", [(1, 1), (2, 15), (3, 16), (13, 17), (16, 33), (17, 31), (18, 1), (30, 50), (31, 16),
                                  (32, 17)])
def test_sizes(monkeypatch, ne, W):
    _compare(monkeypatch, _molecule(ne), W, 2 * ne + 3, sampling=1, qf_modification=2, refresh_interval=7)


@pytest.mark.parametrize("kw", [dict(sampling=0, qf_modification=0, dt=0.09), dict(sampling=0, qf_modification=1),
                                dict(sampling=1, qf_modification=1, qf_equal_a=0.3),
                                dict(sampling=1, qf_modification=0, exact_single_electron_gf=1),
                                dict(sampling=1, qf_modification=2, exact_single_electron_gf=1, old_walker_acceptance=1)])
def test_vmc_forms(monkeypatch, kw):
    _compare(monkeypatch, make_system("vmc_water_10e", seed=1), 40, 33, first=5, **kw)


@pytest.mark.parametrize("kw", [dict(energy_modification=1, reweighting=2, energy_cutoff=QMCB_ECUT_BDJM_PUSH88),
                                dict(energy_modification=2, reweighting=0, energy_cutoff=QMCB_ECUT_UMRIGAR93),
                                dict(energy_modification=0, reweighting=1, dynamic_time_step=1,
                                     energy_cutoff=QMCB_ECUT_BDJM_PUSH88),
                                dict(energy_modification=1, reweighting=2, walker_deletion=1, reweight_start_step=20,
                                     energy_cutoff=QMCB_ECUT_BDJM_PUSH88)])
def test_dmc_forms(monkeypatch, kw):
    _compare(monkeypatch, make_system("vmc_water_10e", seed=1), 64, 47, run_type=QMCB_DMC, sampling=1, qf_modification=2,
             energy_trial=-20.0, energy_estimated=-20.0, energy_original=-20.0, population_control=100.0,
             refresh_interval=15, **{"reweight_start_step": 0, **kw})


@pytest.mark.parametrize("kind", ["none", "cambridge2", "half"])
def test_correlation_forms(monkeypatch, kind):
    s = _molecule(14, jastrow=kind != "none")
    if kind == "cambridge2":
        s = with_cambridge2(s, seed=3)
    if kind == "half":  # no parallel-spin function
        s = dataclasses.replace(s, ee_para_up=None, ee_para_dn=None)
    _compare(monkeypatch, s, 20, 31, sampling=1, qf_modification=2)
