"""The orbital rows' buffer of the batched FP64 kernel: counted by
qmcb_state_bytes and the server's footprint, and not held by a handle whose moves
all run in the sweep kernel."""
import dataclasses

import pytest

from qmcbeaver_b200.api import QMCB200Functions
from qmcbeaver_b200.desc import QMCB_IMPORTANCE_SAMPLING, QMCB_UMRIGAR93_IMPORTANCE_SAMPLING, run_params
from qmcbeaver_b200.serving import state_footprint
from qmcbeaver_b200.system import make_random_molecule, make_system, with_three_body

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("walkers", [100, 3000])
@pytest.mark.parametrize("form", ["plain", "cusps", "three-body", "34 electrons", "134 electrons"])
def test_footprint_counts_the_rows(form, walkers):
    s = make_system("vmc_water_10e", seed=1)
    if form == "cusps":
        s = dataclasses.replace(s, replace_cusps=True)
    elif form == "three-body":
        s = with_three_body(s, seed=3)
    elif form != "plain":
        ne = int(form.split()[0])
        s = make_random_molecule(ne, ne // 6, 2 * ne, 5.0 + ne / 12, (1, 6, 7, 8), seed=ne)
    f = QMCB200Functions(s, 2 * walkers)
    assert f.state_bytes() == state_footprint(s, walkers)
    f.close()


def test_small_spins_take_the_rows_with_umrigar93_moves():
    s, cap = make_system("dmc_6nuc_30e", seed=1), 8192
    f = QMCB200Functions(s, cap, run_params(sampling=QMCB_IMPORTANCE_SAMPLING, qf_modification=2, dt=0.01))
    alone = f.state_bytes()
    assert alone == cap * 3232 * 8  # the walkers' blocks
    f.set_params(run_params(sampling=QMCB_UMRIGAR93_IMPORTANCE_SAMPLING, qf_modification=2, dt=0.01))
    assert f.state_bytes() == alone + cap * 5 * 15 * 8
    f.set_profiling(True)
    f.init_walkers(s.initial_positions(cap // 2, seed=1))
    f.run_steps(0, 4)
    assert f.kernel_stats()["rows_prep"]["launches"] == 4
    f.close()
