"""Shells that need care in the tables of the batched rows.  Generally
contracted ones listed component by component (px px py py pz pz, several
contractions over the same exponents): the runs that share their exponents then
hold a component twice and lack another, so they are no complete p or d shells.
Shells cut by a chunk's end.  Full evaluations, moves of the sweep kernel and
moves on batched rows against the oracle."""
import dataclasses

import numpy as np
import pytest

from qmcbeaver_b200.system import BasisFunction, make_random_molecule
from test_rows64_gpu import _check, _molecule

pytestmark = pytest.mark.gpu


def _by_component(s, components, n_prim):
    """The molecule with two contractions of each component on its first atom."""
    rng = np.random.default_rng(7)
    exps = np.sort(10.0 ** rng.uniform(-0.7, 1.0, n_prim))[::-1].copy()
    added = [BasisFunction(c, exps.copy(), 0.3 * rng.standard_normal(n_prim)) for c in components for _ in range(2)]
    k0 = len(s.basis[0])
    basis = [list(s.basis[0]) + added] + [list(b) for b in s.basis[1:]]
    mo = np.insert(s.mo, [k0] * len(added), 0.1 * rng.standard_normal((s.mo.shape[0], len(added))), axis=1)
    out = dataclasses.replace(s, basis=basis, mo=mo, name=s.name + " by component")
    out.check_exponent_cache()
    return out


@pytest.mark.parametrize("components", [("px", "py", "pz"), ("dxx", "dyy", "dzz", "dxy", "dxz", "dyz")])
@pytest.mark.parametrize("ne,W", [(3, 1030), (16, 40), (40, 40), (40, 3201)])
def test_components_listed_twice_match_oracle(ne, W, components):
    s = make_random_molecule(ne, max(1, ne // 6), 3 * ne, 5.0 + ne / 12, (1, 6, 7, 8), seed=ne, orbitals="random")
    s = _by_component(s, components, 2 + len(components) // 6)
    _check(s, W, [0, s.n_alpha - 1, ne - 1], np.array([0, W // 2, W - 1]))


# 40 functions a chunk: an f shell and shells of d and p functions are cut by the
# chunks' ends (f 2 + 8, 5 + 5, 4 + 6; d 1 + 5, 2 + 4, 5 + 1; p 1 + 2, 2 + 1)
@pytest.mark.parametrize("ne,nb", [(22, 104), (22, 105), (29, 142), (30, 141)])
def test_shells_cut_by_a_chunks_end_match_oracle(ne, nb):
    s = _molecule(ne, nb, True)
    _check(s, 40, [0, s.n_alpha - 1, s.n_alpha, ne - 1], np.array([0, 15, 16, 39]))
