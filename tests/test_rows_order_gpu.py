"""The rounding of the orbital rows: the batched kernels add the basis
functions' contributions in the functions' order and round every radial sum as
the one-warp-per-walker kernels do, so a walker's results are the same bits
however many walkers are evaluated with it, and as near to the 80-bit values as
a plain sum in that order."""
import dataclasses

import numpy as np
import pytest

from qmcbeaver_b200.api import QMCB200Functions
from qmcbeaver_b200.system import make_random_molecule
from test_rows64_gpu import _odd_shells

pytestmark = pytest.mark.gpu


def _molecule(ne, nb, odd):
    s = make_random_molecule(ne, max(1, ne // 6), nb, 5.0 + ne / 12, (1, 6, 7, 8), seed=ne, orbitals="random")
    return _odd_shells(s) if odd else s


@pytest.mark.parametrize("ne,nb,odd", [(34, 99, False), (47, 150, True), (66, 200, True), (100, 301, False)])
def test_moves_are_the_same_bits_at_any_number_of_walkers(ne, nb, odd):
    # 8 walkers take their rows in the move kernel, 3,201 (more than one wave of
    # it) from the batched kernel
    s = _molecule(ne, nb, odd)
    W, few = 3201, 8
    f = QMCB200Functions(s, W, qf_modification=2, dt=0.01)
    g = QMCB200Functions(s, few, qf_modification=2, dt=0.01)
    R = s.initial_positions(W, seed=4, sigma=0.7)
    rng = np.random.default_rng(5)
    f.evaluate(np.arange(W), R, -1)
    g.evaluate(np.arange(few), R[:few], -1)
    for e in (0, s.n_alpha - 1, ne - 1):
        R[:, e] += 0.2 * rng.standard_normal((W, 3))
        many = f.evaluate(np.arange(W), R, e)
        one = g.evaluate(np.arange(few), R[:few], e)
        for k in one:
            assert np.array_equal(many[k][:few], one[k]), (e, k)
    f.close()
    g.close()


@pytest.mark.parametrize("ne,nb,odd", [(1, 31, False), (2, 60, True), (4, 77, False)])
def test_full_evaluations_are_the_same_bits_at_any_number_of_walkers(ne, nb, odd):
    # up to four electrons a call below 1,024 walkers runs in one kernel
    s = _molecule(ne, nb, odd)
    W, few = 1030, 6
    f = QMCB200Functions(s, W, qf_modification=2, dt=0.01)
    R = s.initial_positions(W, seed=4, sigma=0.7)
    many = f.evaluate(np.arange(W), R, -1)
    one = f.evaluate(np.arange(few), R[:few], -1)
    for k in one:
        if k != "log_abs_psi":  # ln|det| adds its pivots in another order
            assert np.array_equal(many[k][:few], one[k]), k
    f.close()


def _sums(s, R):
    """psi and d psi/dx of one electron at R[walkers][3]: in 80 bits, and in
    FP64 by a plain sum over the functions in their order."""
    atom, powers, nprim, offset, exponent, coefficient = s.flat_basis()
    out = []
    for T in (np.longdouble, np.float64):
        value, slope = np.zeros(len(R), T), np.zeros(len(R), T)
        for k in range(len(atom)):
            x = (R - s.coords[atom[k]]).astype(T)
            a, b, c = (int(p) for p in powers[k])
            E0, E1 = np.zeros(len(R), T), np.zeros(len(R), T)
            for i in range(offset[k], offset[k] + nprim[k]):
                t = T(coefficient[i]) * np.exp(-T(exponent[i]) * (x * x).sum(1))
                E0, E1 = E0 + t, E1 + t * T(exponent[i])
            yz = x[:, 1] ** b * x[:, 2] ** c
            P, Px = x[:, 0] ** a * yz, (a * x[:, 0] ** max(a - 1, 0)) * yz
            value = value + T(s.mo_alpha()[0, k]) * (E0 * P)
            slope = slope + T(s.mo_alpha()[0, k]) * (E0 * Px - 2 * x[:, 0] * P * E1)
        out.append((value, slope))
    return out


def test_rows_are_as_accurate_as_a_sum_in_the_functions_order():
    # One electron, 180 functions on 9 atoms in several chunks: grad = psi_x /
    # psi.  The plain FP64 restatement rounds each product and each sum, the
    # kernel (fused) each sum only, and both share the exponentials' and the
    # polynomials' rounding, so the kernel's median error is no larger; 15 % for
    # the spread of two medians over 4,096 positions.
    s = make_random_molecule(1, 9, 180, 8.0, (1, 6, 7, 8), seed=3, orbitals="random")
    s = dataclasses.replace(s, ee_para_up=None, ee_para_dn=None, ee_anti=None, en_up={}, en_dn={})
    W = 4096
    f = QMCB200Functions(s, W)
    R = s.initial_positions(W, seed=4, sigma=1.0)
    got = f.evaluate(np.arange(W), R, -1)["grad"][:, 0, 0]
    f.close()
    (v, d), (v64, d64) = _sums(s, R[:, 0])
    exact = d / v
    err, plain = (np.abs((x - exact) / exact).astype(float) for x in (got, d64 / v64))
    print("median errors: kernel %.2e, plain sum %.2e" % (np.median(err), np.median(plain)))
    assert np.median(err) <= 1.15 * np.median(plain)
