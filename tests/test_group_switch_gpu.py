"""A group whose members' run parameters change between batches of the same
number of steps: every member follows the chain it follows alone."""
import numpy as np
import pytest

from qmcbeaver_b200.api import QMCB200Group
from qmcbeaver_b200.desc import QMCB_DMC, QMCB_IMPORTANCE_SAMPLING, QMCB_UMRIGAR93_IMPORTANCE_SAMPLING
from qmcbeaver_b200.system import make_random_molecule, with_three_body
from test_group_gpu import _dmc_params, _handles, _params

pytestmark = pytest.mark.gpu


def _systems():
    sizes = [(6, 1, 24, 200), (10, 2, 40, 150), (36, 7, 144, 120)]
    out = [(make_random_molecule(ne, nn, nb, 5.0 + ne / 10, (1, 6, 7, 8), seed=30 + k), w)
           for k, (ne, nn, nb, w) in enumerate(sizes)]
    out[1] = (with_three_body(out[1][0], seed=3), out[1][1])
    return out


def test_vmc_then_dmc_without_refreshes():
    systems = _systems()
    solo, grouped = _handles(systems, _params), _handles(systems, _params)
    g = QMCB200Group(grouped)
    g.set_config(0)
    n = 36
    g.run_steps(0, n)
    for f in solo:
        f.run_steps(0, n)
    for f, h in zip(solo, grouped):
        e0 = float(np.median(f.get_walkers()["e_local"]))
        p = _dmc_params(0, e0)
        p.refresh_interval = 0
        assert p.run_type == QMCB_DMC
        f.set_params(p)
        h.set_params(p)
    got = g.run_steps(n, n)
    for f, h, st_g in zip(solo, grouped, got):
        st = f.run_steps(n, n)
        assert st_g.n_walkers == st.n_walkers
        assert st.final_weight > 0  # the last branching pass's sum
        assert st_g.final_weight == pytest.approx(st.final_weight, rel=1e-9)
        a, b = f.get_walkers(), h.get_walkers()
        assert np.array_equal(a["R"], b["R"])
        assert np.allclose(a["weight"], b["weight"], rtol=1e-9)
    g.close()


def test_sweeping_members_alone_need_no_tuning():
    """Members of small spins run on streams of their own, whatever the launch
    configuration of the others: nothing to try, and nothing of theirs enters
    the kernel statistics of their own calls."""
    systems = [x for k, x in enumerate(_systems()) if k == 0] * 2
    grouped = _handles(systems, _params)
    for f in grouped:
        f.set_profiling(True)
    g = QMCB200Group(grouped)
    g.run_steps(0, 12)
    assert g.config()["chosen"] >= 0
    for f in grouped:
        assert all(v["launches"] == 0 for v in f.kernel_stats().values())
        f.run_steps(12, 3)
        assert f.kernel_stats()["move"]["launches"] == 1
    g.close()


def test_sampling_switched_after_the_group_was_made():
    systems = _systems()
    solo, grouped = _handles(systems, _params), _handles(systems, _params)
    g = QMCB200Group(grouped)
    step = 0
    for sampling in (QMCB_IMPORTANCE_SAMPLING, QMCB_UMRIGAR93_IMPORTANCE_SAMPLING, QMCB_IMPORTANCE_SAMPLING):
        for k, (f, h) in enumerate(zip(solo, grouped)):
            f.set_params(_params(k, sampling))
            h.set_params(_params(k, sampling))
        for _ in range(3):
            g.run_steps(step, 11)
            for f in solo:
                f.run_steps(step, 11)
            step += 11
        for f, h in zip(solo, grouped):
            assert np.array_equal(f.get_walkers()["R"], h.get_walkers()["R"]), sampling
    g.close()
