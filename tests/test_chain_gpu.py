"""Metropolis chains of small spins against walkers recorded from the
one-warp-per-walker kernel (golden/make_chains.py): the sweep kernel rounds every
number that the chain goes on from -- rows, inverses, ratio sums, pair sums,
drifts -- as that kernel does, so the walkers are the same bits after any number
of moves, also where a walker next to a node would amplify a rounding."""
import os
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, os.path.join(HERE, "golden"))
from make_chains import CHAINS, run  # noqa: E402

pytestmark = pytest.mark.gpu
GOLDEN = np.load(os.path.join(HERE, "golden", "chains", "small_spins.npz"))


@pytest.mark.parametrize("name", list(CHAINS))
def test_walkers_are_the_recorded_ones(name):
    got = run(name)
    want = {k: GOLDEN[f"{name}.{k}"] for k in got}
    assert np.array_equal(got["R"], want["R"])
    assert np.array_equal(got["sign"], want["sign"])
    # the sums over a walker's columns and determinants add in another order:
    # some roundings of terms up to 1e3 times the local energy
    for k in ("e_local", "log_abs_psi"):
        assert np.max(np.abs(got[k] - want[k]) / np.maximum(np.abs(want[k]), 1.0)) < 1e-12, k
