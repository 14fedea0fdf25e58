"""The batched FP64 orbital rows (32 walkers per CTA, FP64 tensor pipe): full
evaluations of all electrons and single-electron moves of more walkers than
one wave of the fused move kernel holds, against the oracle at the sizes where
its tiling changes (8-orbital tiles, one or two warps per 16-row tile, orbital
splits, partly filled walker tiles and chunks) and on shells that take its
general path (f functions, lone members, more than three primitives)."""
import dataclasses

import numpy as np
import pytest

from helpers import PARITY_RTOL, compare, cond_bounds, slater_conditions
from qmcbeaver_b200.api import QMCB200Functions
from qmcbeaver_b200.system import BasisFunction, make_random_molecule

pytestmark = pytest.mark.gpu


def _odd_shells(s):
    """The molecule with an f shell, a lone dxy of four primitives, an s of six
    and a p pair added on its first atom."""
    rng = np.random.default_rng(3)
    new = [("f" + t, 2) for t in ("xxx", "yyy", "zzz", "xxy", "xxz", "yyx", "yyz", "zzx", "zzy", "xyz")]
    new += [("dxy", 4), ("s", 6), ("px", 3), ("pz", 3)]
    exps = {n: np.sort(10.0 ** rng.uniform(-0.7, 1.0, n))[::-1].copy() for n in (2, 3, 4, 6)}
    added = [BasisFunction(t, exps[n].copy(), 0.3 * rng.standard_normal(n)) for t, n in new]
    basis = [list(s.basis[0]) + added] + [list(b) for b in s.basis[1:]]
    k0 = len(s.basis[0])
    mo = np.insert(s.mo, [k0] * len(added), 0.1 * rng.standard_normal((s.mo.shape[0], len(added))), axis=1)
    out = dataclasses.replace(s, basis=basis, mo=mo, name=s.name + " odd shells")
    out.check_exponent_cache()
    return out


def _molecule(ne, nb, odd):
    s = make_random_molecule(ne, max(1, ne // 6), nb, 5.0 + ne / 12, (1, 6, 7, 8), seed=ne, orbitals="random")
    return _odd_shells(s) if odd else s


def _check(s, W, electrons, watched):
    from oracle.evaluators import OracleEvaluator
    orc = OracleEvaluator(s, qf_mod=2, dt=0.01)
    f = QMCB200Functions(s, W, qf_modification=2, dt=0.01)
    ws = orc.new_walkers(len(watched))
    R = s.initial_positions(W, seed=4, sigma=0.7)
    rng = np.random.default_rng(5)
    slope, limit = cond_bounds(s)
    worst = np.zeros(len(watched))
    for e in [-1] + list(electrons):
        if e >= 0:
            R[:, e] += 0.2 * rng.standard_normal((W, 3))
        out = {k: v[watched] for k, v in f.evaluate(np.arange(W), R, e).items()}
        orc.evaluate(ws, R[watched], e)
        ref = orc.results(ws)
        worst = np.maximum(worst, slater_conditions(orc, ws, s))
        # E_L = -lap/2 + V cancels; its rounding scales with the terms
        amp = (np.abs(ref["lap"]) / 2 + np.abs(ref["potential"])) / np.maximum(np.abs(ref["e_local"]), 1.0)
        for i in range(len(watched)):
            one = np.arange(len(watched)) == i
            compare(out, ref, max(PARITY_RTOL, slope * worst[i]) if worst[i] >= limit else PARITY_RTOL,
                    f"{s.name} electron {e} walker {watched[i]} (cond {worst[i]:.1e})", mask=one, kappa=amp)
    f.close()


@pytest.mark.parametrize("ne,nb,W,odd", [(1, 4, 1, False), (3, 9, 33, False), (16, 47, 32, False), (18, 48, 31, True),
                                         (33, 99, 65, False), (64, 193, 34, False), (66, 200, 33, True),
                                         (130, 265, 33, False)])
def test_full_evaluation_matches_oracle(ne, nb, W, odd):
    _check(_molecule(ne, nb, odd), W, [], np.unique([0, W // 2, W - 1]))


@pytest.mark.parametrize("ne,nb,odd", [(3, 9, False), (16, 49, True), (18, 48, False), (66, 200, True),
                                       (130, 265, False)])
def test_moves_of_many_walkers_match_oracle(ne, nb, odd):
    s = _molecule(ne, nb, odd)
    W = 3201  # more than 148 SMs hold of any molecule; the last tile holds one walker
    _check(s, W, [0, s.n_alpha - 1, ne - 1, 0], np.array([0, 31, 32, 1777, 3199, 3200]))


def test_moves_of_disjoint_walkers_on_two_streams_match_oracle():
    # evaluate_device on two callers' streams, half of the walkers each: the
    # calls may overlap, so nothing but the walkers' own state may be written
    import ctypes
    import torch
    from oracle.evaluators import OracleEvaluator
    s, W, watched = _molecule(130, 265, False), 1024, np.array([0, 511, 512, 1023])
    orc = OracleEvaluator(s, qf_mod=2, dt=0.01)
    f = QMCB200Functions(s, W, qf_modification=2, dt=0.01)
    ws = orc.new_walkers(len(watched))
    R = s.initial_positions(W, seed=4, sigma=0.7)
    f.evaluate(np.arange(W), R, -1)
    orc.evaluate(ws, R[watched], -1)
    worst = slater_conditions(orc, ws, s)
    rng = np.random.default_rng(5)
    streams = [torch.cuda.Stream() for _ in range(2)]
    slots = torch.arange(W, dtype=torch.int32, device="cuda")
    sides = []
    for e in (0, 64, 65, 129):
        R[:, e] += 0.2 * rng.standard_normal((W, 3))
        out = [torch.zeros(W * k, dtype=torch.float64, device="cuda") for k in (1, 1, 390, 390, 1, 1, 3)]
        sides.append((e, torch.tensor(R, device="cuda"), out, torch.zeros(W, dtype=torch.uint8, device="cuda")))
        orc.evaluate(ws, R[watched], e)
        worst = np.maximum(worst, slater_conditions(orc, ws, s))
    torch.cuda.synchronize()
    for e, r, out, status in sides:
        for half, st in enumerate(streams):
            at = half * (W // 2)
            args = [ctypes.c_void_p(x.data_ptr() + at * x.element_size() * (x.numel() // W)) for x in out + [status]]
            rc = f.lib.qmcb_evaluate_device(f.h, e, ctypes.c_void_p(slots.data_ptr() + 4 * at), W // 2,
                                            ctypes.c_void_p(r.data_ptr() + 8 * 390 * at), *args,
                                            ctypes.c_void_p(st.cuda_stream))
            assert rc == 0
    torch.cuda.synchronize()
    ref = orc.results(ws)
    slope, limit = cond_bounds(s)
    names = ("log_abs_psi", "sign", "grad", "mod_grad", "lap", "e_local")
    out = {k: v.cpu().numpy().reshape(W, -1)[watched].reshape(np.shape(ref[k])) for k, v in zip(names, sides[-1][2])}
    out["potential"] = sides[-1][2][-1].cpu().numpy().reshape(W, 3)[watched, 0]
    amp = (np.abs(ref["lap"]) / 2 + np.abs(ref["potential"])) / np.maximum(np.abs(ref["e_local"]), 1.0)
    for i in range(len(watched)):
        one = np.arange(len(watched)) == i
        compare(out, ref, max(PARITY_RTOL, slope * worst[i]) if worst[i] >= limit else PARITY_RTOL,
                f"walker {watched[i]} (cond {worst[i]:.1e})", mask=one, kappa=amp)
    f.close()
