"""The calls whose speed matters to a user of qmcbeaver_b200, through its public
entry points: a driver that evaluates walkers it owns (``evaluate``,
``evaluate_moved``, ``qmcb_evaluate_device``), Metropolis / DMC blocks on
device-resident walkers (``run_steps``) and several molecules stepped as one
group (``QMCB200Group``).

``listed`` gives the cases, ``draw`` others of the same ranges, ``prepare``
what a program holds before the call, ``run`` one pass, ``work`` the bytes and
operations it cannot do without, ``exact`` the evaluations' values in plain
torch double precision.  The Markov-chain passes have no value that plain
torch could give (their proposals come from the library's random streams).
"""
import ctypes
import dataclasses
import functools
import math

import numpy as np
import torch

from qmcbeaver_b200.api import OUT_ALL, QMCB200Functions, QMCB200Group
from qmcbeaver_b200.desc import (QMCB_DMC, QMCB_ECUT_BDJM_PUSH88, QMCB_EMOD_UMRIGAR93, QMCB_IMPORTANCE_SAMPLING,
                                 QMCB_NO_IMPORTANCE_SAMPLING, QMCB_PREC_FP64, QMCB_PREC_INT8_SLICES,
                                 QMCB_QF_NONE, QMCB_QF_UMRIGAR93_UNEQUAL, QMCB_UMRIGAR93_IMPORTANCE_SAMPLING,
                                 QMCB_VMC, run_params)
from qmcbeaver_b200.system import make_random_molecule, make_system, with_cambridge2, with_determinants, with_three_body

SAMPLING = {"metropolis": QMCB_NO_IMPORTANCE_SAMPLING, "drift": QMCB_IMPORTANCE_SAMPLING,
            "umrigar93": QMCB_UMRIGAR93_IMPORTANCE_SAMPLING}
PRECISION = {"fp64": QMCB_PREC_FP64, "int8": QMCB_PREC_INT8_SLICES}
REFRESH = 50  # moves between refreshes of the inverses, as bench.py runs


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # one walker of the water workload evaluated afresh: a driver that
        # adds a walker, and the latency of the host path
        {"name": "evaluate-water-1", "kind": "evaluate", "molecule": "vmc_water_10e", "walkers": 1},
        # walker initialisation and all-electron moves of a medium molecule
        # from host arrays
        {"name": "evaluate-30e-4096", "kind": "evaluate", "molecule": "dmc_6nuc_30e", "walkers": 4096},
        # a host driver moving one electron at a time (the drop-in for
        # QMCFunctions::evaluate), outputs in page-locked memory
        {"name": "moved-30e-4096", "kind": "moved", "molecule": "dmc_6nuc_30e", "walkers": 4096},
        # the same for a driver whose walkers live on the device; an odd
        # electron count, spins beyond one warp's lanes
        {"name": "device-71e-1024", "kind": "device", "molecule": "core", "electrons": 71, "walkers": 1024},
        # the reference's smallest standard run: 100 walkers of water, plain
        # Metropolis; launches and latency
        {"name": "vmc-water-100", "kind": "chain", "run": "vmc", "molecule": "vmc_water_10e", "walkers": 100,
         "steps": 50, "sampling": "metropolis", "precision": "fp64"},
        # the headline benchmark: one DMC block of 150 moves, five branching
        # passes, three refreshes
        {"name": "dmc-30e-16384", "kind": "chain", "run": "dmc", "molecule": "dmc_6nuc_30e", "walkers": 16384,
         "steps": 150, "sampling": "drift", "precision": "fp64"},
        # one DMC sweep of the large molecule in plain FP64, and with its
        # orbital rows from the int8 tensor-core contraction (the reduced
        # modes below FP64 accuracy miss the energy tolerance and are for study)
        {"name": "dmc-100e-8192", "kind": "chain", "run": "dmc", "molecule": "mixed_20nuc_100e", "walkers": 8192,
         "steps": 100, "sampling": "drift", "precision": "fp64"},
        {"name": "dmc-100e-8192-int8", "kind": "chain", "run": "dmc", "molecule": "mixed_20nuc_100e",
         "walkers": 8192, "steps": 100, "sampling": "drift", "precision": "int8"},
        # the reference's default sampling with everything its inputs switch
        # on: cusp replacement, Cambridge two- and three-body Jastrows
        {"name": "umrigar-16e-4096", "kind": "chain", "run": "vmc", "molecule": "vmc_threebody_16e",
         "cusps": True, "walkers": 4096, "steps": 48, "sampling": "umrigar93", "precision": "fp64"},
        # a CI expansion of twelve determinants
        {"name": "multidet-12e-4096", "kind": "chain", "run": "vmc", "molecule": "vmc_multidet_12e",
         "walkers": 4096, "steps": 48, "sampling": "drift", "precision": "fp64"},
        # many small jobs on one GPU: twelve molecules of 4 to 40 electrons,
        # 256 to 2,048 walkers each, stepped together
        {"name": "group-12", "kind": "group", "members": 12, "steps": 40, "molecules": 29},
        # the largest molecule of the uneven-batching workload
        {"name": "vmc-196e-512", "kind": "chain", "run": "vmc", "molecule": "random", "electrons": 196,
         "walkers": 512, "steps": 100, "sampling": "drift", "precision": "fp64"},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["evaluate", "moved", "device", "vmc", "vmc", "dmc", "dmc", "int8", "features", "multidet",
                       "group"])
    if kind in ("evaluate", "moved", "device"):
        case = {"kind": kind, "molecule": "core", "electrons": _log_int(rng, 3, 80),
                "walkers": _log_int(rng, 1, 4096)}
    elif kind in ("vmc", "dmc", "int8"):
        case = {"kind": "chain", "run": "vmc" if kind == "vmc" else "dmc",
                "molecule": "core", "electrons": _log_int(rng, 4 if kind == "vmc" else 12, 80),
                "walkers": _log_int(rng, 64, 16384), "steps": rng.randint(20, 150),
                "sampling": rng.choice(["metropolis", "drift"]) if kind == "vmc" else "drift",
                "precision": "int8" if kind == "int8" else "fp64"}
    elif kind == "features":
        case = {"kind": "chain", "run": "vmc", "molecule": "features", "cusps": rng.random() < 0.5,
                "electrons": rng.randint(4, 24), "walkers": _log_int(rng, 64, 8192), "steps": rng.randint(16, 64),
                "sampling": rng.choice(["drift", "umrigar93"]), "precision": "fp64"}
    elif kind == "multidet":
        case = {"kind": "chain", "run": "vmc", "molecule": "multidet", "electrons": rng.randint(4, 16),
                "determinants": rng.randint(9, 16), "walkers": _log_int(rng, 64, 8192),
                "steps": rng.randint(16, 64), "sampling": "drift", "precision": "fp64"}
    else:
        case = {"kind": "group", "members": rng.randint(2, 12), "steps": rng.randint(20, 60),
                "molecules": rng.randint(100, 10 ** 6)}
    # no dearer than the listed ones
    dearest = max(work(c)["flops"] for c in listed()) / 2
    while kind != "group" and case["walkers"] > 1 and work(case)["flops"] > dearest:
        case["walkers"] = case["walkers"] // 2 + 1
    return case


# ---------------------------------------------------------------- molecules
def _random_molecule(electrons, orbitals, seed):
    # the serving and batching workloads' shape: one nucleus per five
    # electrons, four basis functions per electron
    nuclei = max(1, electrons // 5)
    box = 2.0 + 3.0 * nuclei ** (1.0 / 3.0)
    return make_random_molecule(electrons, nuclei, 4 * electrons, box, (1, 6, 7, 8), seed=seed, min_sep=1.4,
                                orbitals=orbitals)


@functools.lru_cache(maxsize=None)
def _molecule(molecule, electrons, cusps, determinants):
    if molecule in ("core", "random"):
        s = _random_molecule(electrons, molecule, electrons)
    elif molecule == "features":
        s = with_three_body(with_cambridge2(_random_molecule(electrons, "core", electrons), seed=2), seed=4)
    elif molecule == "multidet":
        s = with_determinants(_random_molecule(electrons, "core", electrons), determinants, 4, seed=3)
    else:
        s = make_system(molecule, seed=1)
    return dataclasses.replace(s, replace_cusps=True) if cusps else s


def _system(case):
    return _molecule(case["molecule"], case.get("electrons", 0), case.get("cusps", False),
                     case.get("determinants", 0))


@functools.lru_cache(maxsize=None)
def _group_plan(molecules, members):
    rng = np.random.default_rng(molecules)
    return [(2 * int(rng.integers(2, 21)), int(rng.integers(256, 2049))) for _ in range(members)]


# ---------------------------------------------------------------- the state
def _params(case, seed):
    metropolis = case.get("sampling") == "metropolis"
    return run_params(sampling=SAMPLING[case.get("sampling", "drift")],
                      qf_modification=QMCB_QF_NONE if metropolis else QMCB_QF_UMRIGAR93_UNEQUAL,
                      dt=0.09 if metropolis else 0.01, refresh_interval=REFRESH, seed=seed + 1, rel_cutoff=0.0,
                      precision=PRECISION[case.get("precision", "fp64")])


def _dmc_params(case, seed, energy, start):
    return run_params(run_type=QMCB_DMC, sampling=QMCB_IMPORTANCE_SAMPLING,
                      qf_modification=QMCB_QF_UMRIGAR93_UNEQUAL, energy_modification=QMCB_EMOD_UMRIGAR93, dt=0.01,
                      refresh_interval=REFRESH, reweight_start_step=start, energy_trial=energy,
                      energy_estimated=energy, energy_original=energy, seed=seed + 1,
                      energy_cutoff=QMCB_ECUT_BDJM_PUSH88, population_control=100.0, walker_deletion=1,
                      precision=PRECISION[case["precision"]])


def _positions(case, seed):
    return _system(case).initial_positions(case["walkers"], seed=seed + 1)


def _condition(s, R):
    """The larger condition number (Frobenius norms) of each walker's two Slater matrices."""
    W, worst = R.shape[0], torch.zeros(R.shape[0], dtype=R.dtype, device=R.device)
    for base, n, mo in ((0, s.n_alpha, s.mo_alpha()), (s.n_alpha, s.n_beta, s.mo_beta())):
        if n:
            C = torch.from_numpy(mo).to(R.device).T
            D = (_basis_rows(s, R[:, base:base + n].reshape(-1, 3), values_only=True)[0] @ C).reshape(W, n, n)
            worst = torch.maximum(worst, D.norm(dim=(1, 2)) * torch.linalg.inv(D).norm(dim=(1, 2)))
    return worst


def _away_from_nodes(case, *configurations):
    """The walkers (of twice as many) that a driver's equilibrated ensemble
    would hold: |psi|^2 keeps it away from the nodes, so the half whose Slater
    matrices are better conditioned in every one of the configurations."""
    s, device = _system(case), "cuda" if torch.cuda.is_available() else "cpu"
    chunk = max(1, int(4e8 // (s.n_electrons * s.n_basis * 8)))
    worst = None
    for R in configurations:
        c = torch.cat([_condition(s, torch.from_numpy(R[i:i + chunk]).to(device)) for i in range(0, len(R), chunk)])
        worst = c if worst is None else torch.maximum(worst, c)
    keep = torch.sort(torch.argsort(worst, stable=True)[:case["walkers"]]).values.cpu().numpy()
    return [np.ascontiguousarray(R[keep]) for R in configurations]


def _evaluated_positions(case, seed):
    return _away_from_nodes(case, _positions(dict(case, walkers=2 * case["walkers"]), seed))[0]


# single-electron calls of one pass: two electrons of each spin, in turn
def _moved_electrons(system):
    first, beta = [0, system.n_alpha // 2], [system.n_alpha, system.n_electrons - 1]
    return [e for e in dict.fromkeys(first + beta) if e < system.n_electrons]


def _move_targets(case, seed):
    """The start R0 and the configurations after each call of an even pass
    (the electrons leave R0) and of an odd one (they go back)."""
    s, W = _system(case), 2 * case["walkers"]
    R0 = _positions(dict(case, walkers=W), seed)
    rng = np.random.default_rng(seed + 77)
    out, R = [], R0
    es = _moved_electrons(s)
    for e in es:
        R = R.copy()
        R[:, e] += 0.2 * rng.standard_normal((W, 3))
        out.append(R)
    R0, *out = _away_from_nodes(case, R0, *out)
    R = out[-1]
    back = []
    for e in es:
        R = R.copy()
        R[:, e] = R0[:, e]
        back.append(R)
    return R0, es, [out, back]


def _pinned(n_electrons, walkers):
    def array(*shape, dtype=torch.float64):
        return torch.zeros(shape, dtype=dtype, pin_memory=True).numpy()
    return dict(log_abs_psi=array(walkers), sign=array(walkers), grad=array(walkers, n_electrons, 3),
                mod_grad=array(walkers, n_electrons, 3), lap=array(walkers), e_local=array(walkers),
                pe=array(walkers, 3), status=array(walkers, dtype=torch.uint8))


OUTPUTS = ("log_abs_psi", "sign", "grad", "mod_grad", "lap", "e_local", "pe", "status")


def prepare(case, seed):
    if case["kind"] == "group":
        return _prepare_group(case, seed)
    s, W = _system(case), case["walkers"]
    if case["kind"] == "evaluate":
        return {"kind": "evaluate", "f": QMCB200Functions(s, W, _params(case, seed)), "slots": np.arange(W),
                "R": _evaluated_positions(case, seed)}
    if case["kind"] in ("moved", "device"):
        R0, es, targets = _move_targets(case, seed)
        f = QMCB200Functions(s, W, _params(case, seed))
        f.evaluate(np.arange(W), R0, -1)
        state = {"kind": case["kind"], "f": f, "electrons": es, "passes": 0, "slots": np.arange(W, dtype=np.int32)}
        if case["kind"] == "moved":
            state["r"] = [[torch.from_numpy(np.ascontiguousarray(R[:, e])).pin_memory().numpy()
                           for e, R in zip(es, side)] for side in targets]
            state["out"] = [_pinned(s.n_electrons, W) for _ in es]
        else:
            state["slots"] = torch.arange(W, dtype=torch.int32, device="cuda")
            state["r"] = [[torch.from_numpy(R).cuda() for R in side] for side in targets]
            N = s.n_electrons

            def buffer(*shape, dtype=torch.float64):
                return torch.zeros(shape, dtype=dtype, device="cuda")
            state["out"] = [dict(log_abs_psi=buffer(W), sign=buffer(W), grad=buffer(W, N, 3),
                                 mod_grad=buffer(W, N, 3), lap=buffer(W), e_local=buffer(W), pe=buffer(W, 3),
                                 status=buffer(W, dtype=torch.uint8)) for _ in es]
            torch.cuda.synchronize()
        return state
    # a chain on equilibrated walkers
    N = s.n_electrons
    if case["run"] == "vmc":
        f = QMCB200Functions(s, W, _params(case, seed))
        f.init_walkers(_positions(case, seed))
        f.run_steps(0, 2 * N)
        return {"kind": "chain", "f": f, "step": 2 * N, "steps": case["steps"], "saved": W}
    f = QMCB200Functions(s, 2 * W, _dmc_params(case, seed, -1.0, 10 ** 9))
    f.init_walkers(_positions(case, seed))
    f.run_steps(0, 2 * N)
    w = f.get_walkers()
    f.set_params(_dmc_params(case, seed, float(np.mean(w["e_local"])), 0))
    f.init_walkers(w["R"])
    f.run_steps(0, N)
    # the population breathes: after each block the program saves three
    # quarters of its target number of walkers
    return {"kind": "chain", "f": f, "step": N, "steps": case["steps"], "saved": 3 * W // 4}


def _prepare_group(case, seed):
    handles, starts = [], []
    for i, (electrons, walkers) in enumerate(_group_plan(case["molecules"], case["members"])):
        s = _molecule("core", electrons, False, 0)
        f = QMCB200Functions(s, walkers, _params({}, seed + 1000 * i))
        starts.append(s.initial_positions(walkers, seed=seed + 1000 * i + 1))
        f.init_walkers(starts[-1])
        handles.append(f)
    g = QMCB200Group(handles)
    step = 0
    while g.config()["chosen"] < 0 and step < 100 * case["steps"]:  # its launch shapes are tuned on real steps
        g.run_steps(step, case["steps"])
        step += case["steps"]
    for f, R in zip(handles, starts):
        f.init_walkers(R)
    g.run_steps(0, case["steps"])
    return {"kind": "group", "group": g, "members": handles, "step": case["steps"], "steps": case["steps"]}


# ---------------------------------------------------------------- one pass
def _stats(st):
    return [st.sum_weight, st.sum_weight_energy, st.sum_weight_energy2, st.sum_accept, st.n_moves, st.final_weight,
            int(st.n_walkers), int(st.n_singular)]


def run(state):
    if state["kind"] == "evaluate":
        out = state["f"].evaluate(state["slots"], state["R"], -1)
        return {k: out[k] for k in OUTPUTS}
    if state["kind"] == "moved":
        side = state["r"][state["passes"] % 2]
        state["passes"] += 1
        for e, r, out in zip(state["electrons"], side, state["out"]):
            state["f"].evaluate_moved(state["slots"], r, e, OUT_ALL, out)
        return state["out"]
    if state["kind"] == "device":
        side = state["r"][state["passes"] % 2]
        state["passes"] += 1
        f, slots = state["f"], state["slots"]
        for e, r, out in zip(state["electrons"], side, state["out"]):
            rc = f.lib.qmcb_evaluate_device(f.h, e, ctypes.c_void_p(slots.data_ptr()), slots.numel(),
                                            ctypes.c_void_p(r.data_ptr()),
                                            *[ctypes.c_void_p(out[k].data_ptr()) for k in OUTPUTS], None)
            if rc != 0:
                raise RuntimeError(f.lib.qmcb_last_error(f.h).decode())
        return state["out"]
    if state["kind"] == "group":
        stats = state["group"].run_steps(state["step"], state["steps"])
        state["step"] += state["steps"]
        walkers = [f.get_walkers() for f in state["members"]]
        return {"stats": np.array([_stats(st) for st in stats]), "R": [w["R"] for w in walkers],
                "e_local": [w["e_local"] for w in walkers], "log_abs_psi": [w["log_abs_psi"] for w in walkers]}
    stats = state["f"].run_steps(state["step"], state["steps"])
    state["step"] += state["steps"]
    out = state["f"].get_walkers(min(state["saved"], int(stats.n_walkers)))
    short = state["saved"] - len(out["weight"])
    if short > 0:
        out = {k: np.concatenate([v, np.zeros((short,) + v.shape[1:])]) for k, v in out.items()}
    out["stats"] = _stats(stats)
    return out


# ---------------------------------------------------------------- its least work
def _sizes(case):
    """(electrons, alpha, beta, basis functions, nuclei, determinants) without building the molecule."""
    known = {"vmc_water_10e": (10, 24, 3, 1), "dmc_6nuc_30e": (30, 120, 6, 1), "mixed_20nuc_100e": (100, 400, 20, 1),
             "vmc_threebody_16e": (16, 64, 4, 1), "vmc_multidet_12e": (12, 48, 3, 12)}
    if case["molecule"] in known:
        N, K, M, D = known[case["molecule"]]
    else:
        N = case["electrons"]
        K, M, D = 4 * N, max(1, N // 5), case.get("determinants", 1)
    return N, N - N // 2, N // 2, K, M, D


def _move_flops(N, n, K, M, D, three_body=False):
    """One single-electron move: basis values and derivatives (about 60
    operations a function), five orbital rows, Sherman-Morrison update and
    ratio sums of the moved spin's determinants, pair terms (about 60 a pair,
    old and new; a three-body term about 600)."""
    return (60 * K + 10 * K * n + D * (4 * n * n + 2 * n) + D * 8 * n * n + 2 * 60 * (N + M) + 40 * N
            + (2 * 600 * N * M if three_body else 0))


def _state_bytes(N, na, nb, D):
    """A walker's positions, gradients, Slater values, derivative rows and inverses."""
    return 8 * (12 * N + sum((5 + D) * n * n for n in (na, nb)))


def _chain_work(N, na, nb, K, M, D, walkers, steps, three_body):
    move = (na * _move_flops(N, na, K, M, D, three_body) + nb * _move_flops(N, nb, K, M, D, three_body)) / N
    refresh = steps / REFRESH * 2 * (na ** 3 + nb ** 3)
    return {"bytes": walkers * (2 * _state_bytes(N, na, nb, D) + 8 * (3 * N + 4)),
            "flops": walkers * (steps * move + refresh)}


def work(case):
    if case["kind"] == "group":
        total = {"bytes": 0.0, "flops": 0.0}
        for electrons, walkers in _group_plan(case["molecules"], case["members"]):
            w = _chain_work(electrons, electrons // 2, electrons // 2, 4 * electrons, max(1, electrons // 5), 1,
                            walkers, case["steps"], False)
            total = {k: total[k] + w[k] for k in total}
        return total
    N, na, nb, K, M, D = _sizes(case)
    W = case["walkers"]
    outputs = 8 * (6 * N + 7) + 1
    if case["kind"] == "evaluate":
        # the state written, positions in, outputs out; basis and rows of
        # every electron, the inverses, the ratio sums, all pairs
        flops = sum(n * (60 * K + 10 * K * n) + 2 * n ** 3 + 8 * n * n for n in (na, nb)) + 60 * N * (N / 2 + M)
        return {"bytes": W * (_state_bytes(N, na, nb, D) + 24 * N + outputs), "flops": W * flops}
    if case["kind"] in ("moved", "device"):
        # the moved spin's inverse read and written, its derivative rows
        # read, the per-electron arrays, a position in, the outputs out
        calls = len({0, (N - N // 2) // 2, na, N - 1})
        one = (8 * (6 * na * na + 5 * na + 12 * N) + outputs + 24, _move_flops(N, na, K, M, D))
        return {"bytes": W * calls * one[0], "flops": W * calls * one[1]}
    three_body = case["molecule"] in ("vmc_threebody_16e", "features")
    return _chain_work(N, na, nb, K, M, D, W, case["steps"], three_body)


# ---------------------------------------------------------------- its exact value
def _pair(fn, r):
    """u, u', u'' of a r / (1 + b r)."""
    a, b = float(fn.num[1]), float(fn.den[1])
    q = 1.0 / (1.0 + b * r)
    return a * r * q, a * q * q, -2.0 * a * b * q ** 3


def _basis_rows(s, r, values_only=False):
    """Values, gradients and Laplacians [5][points][K] of the basis at r[points][3] (or [1][points][K])."""
    atom, powers, nprim, offset, exponent, coefficient = s.flat_basis()
    dev, P = r.device, int(nprim.max())
    K = len(atom)
    al, co = np.zeros((K, P)), np.zeros((K, P))
    for k in range(K):
        al[k, :nprim[k]] = exponent[offset[k]:offset[k] + nprim[k]]
        co[k, :nprim[k]] = coefficient[offset[k]:offset[k] + nprim[k]]
    al, co = torch.from_numpy(al).to(dev), torch.from_numpy(co).to(dev)
    pw = torch.from_numpy(powers.astype(np.int64)).to(dev)
    x = r[:, None, :] - torch.from_numpy(s.coords[atom]).to(dev)[None]
    r2 = (x * x).sum(-1)
    E0, E1, E2 = (torch.zeros_like(r2) for _ in range(3))
    for i in range(P):
        t = co[:, i] * torch.exp(-al[:, i] * r2)
        E0, E1, E2 = E0 + t, E1 + t * al[:, i], E2 + t * al[:, i] ** 2

    def power(d, less):
        p = pw[:, d] - less
        return torch.where(p >= 0, x[..., d] ** p.clamp(min=0).to(x.dtype), torch.zeros_like(r2))
    p0, p1, p2 = ([power(d, less) for d in range(3)] for less in range(3))
    n = [pw[:, d].to(x.dtype) for d in range(3)]
    poly = p0[0] * p0[1] * p0[2]
    rows = [E0 * poly]
    if values_only:
        return torch.stack(rows)
    lap = torch.zeros_like(r2)
    for d in range(3):
        others = p0[(d + 1) % 3] * p0[(d + 2) % 3]
        rows.append(E0 * n[d] * p1[d] * others - 2.0 * E1 * x[..., d] * poly)
        lap = lap + E0 * n[d] * (n[d] - 1) * p2[d] * others
    rows.append(lap + poly * (4.0 * r2 * E2 - (4.0 * pw.sum(-1).to(x.dtype) + 6.0) * E1))
    return torch.stack(rows)


def _evaluate_exact(s, R, dt, modified):
    """log|psi|, sign, drift, modified drift, lap(psi)/psi, E_L and potentials of R[walkers][N][3]."""
    W, N = R.shape[0], R.shape[1]
    dev = R.device
    log_psi, sign = torch.zeros(W, dtype=R.dtype, device=dev), torch.ones(W, dtype=R.dtype, device=dev)
    grad_D, lap_D = torch.zeros_like(R), torch.zeros(W, dtype=R.dtype, device=dev)
    for base, n, mo in ((0, s.n_alpha, s.mo_alpha()), (s.n_alpha, s.n_beta, s.mo_beta())):
        if n == 0:
            continue
        C = torch.from_numpy(mo).to(dev).T
        rows = _basis_rows(s, R[:, base:base + n].reshape(-1, 3)) @ C
        rows = rows.reshape(5, W, n, n)  # [quantity][walker][electron][orbital]
        sg, ld = torch.linalg.slogdet(rows[0])
        inverse = torch.linalg.inv(rows[0]).transpose(1, 2)
        log_psi, sign = log_psi + ld, sign * sg
        for d in range(3):
            grad_D[:, base:base + n, d] = (rows[1 + d] * inverse).sum(-1)
        lap_D = lap_D + (rows[4] * inverse).sum((1, 2))
    nuc, Z = torch.from_numpy(s.coords).to(dev), torch.from_numpy(np.asarray(s.Z, np.float64)).to(dev)
    U, U_lap, U_grad = torch.zeros_like(log_psi), torch.zeros_like(log_psi), torch.zeros_like(R)
    ee, en = torch.zeros_like(log_psi), torch.zeros_like(log_psi)
    for i in range(N):
        for j in range(i):
            v = R[:, i] - R[:, j]
            r = v.norm(dim=-1)
            ee = ee + 1.0 / r
            up = (i < s.n_alpha, j < s.n_alpha)
            u, du, d2u = _pair(s.ee_anti if up[0] != up[1] else s.ee_para_up if up[0] else s.ee_para_dn, r)
            g = (du / r)[:, None] * v
            U, U_lap = U + u, U_lap + 2.0 * (2.0 * du / r + d2u)
            U_grad[:, i] += g
            U_grad[:, j] -= g
        for A, label in enumerate(s.labels):
            v = R[:, i] - nuc[A]
            r = v.norm(dim=-1)
            en = en - Z[A] / r
            u, du, d2u = _pair((s.en_up if i < s.n_alpha else s.en_dn)[label], r)
            U, U_lap = U + u, U_lap + 2.0 * du / r + d2u
            U_grad[:, i] += (du / r)[:, None] * v
    grad = grad_D + U_grad
    lap = lap_D + U_lap + (U_grad * (2.0 * grad_D + U_grad)).sum((1, 2))
    nn = sum(float(s.Z[a] * s.Z[b]) / float(np.linalg.norm(s.coords[a] - s.coords[b]))
             for a in range(len(Z)) for b in range(a))
    potential = nn + ee + en
    mod = grad
    if modified:
        # each electron's drift limited as Umrigar, Nightingale and Runge (1993)
        v = R[:, :, None, :] - nuc
        near = (v * v).sum(-1).argmin(-1)
        v = torch.gather(v, 2, near[:, :, None, None].expand(-1, -1, 1, 3))[:, :, 0]
        d2, g2 = (v * v).sum(-1), (grad * grad).sum(-1)
        t = Z[near] ** 2 * d2
        a = 0.5 * (1.0 + (v * grad).sum(-1) / (d2 * g2).sqrt()) + t / (10.0 * (4.0 + t))
        mod = grad * ((-1.0 + (1.0 + 2.0 * a * g2 * dt).sqrt()) / (a * g2 * dt))[..., None]
    return {"log_abs_psi": log_psi + U, "sign": sign, "grad": grad, "mod_grad": mod, "lap": lap,
            "e_local": -0.5 * lap + potential, "pe": torch.stack([potential, en, ee], 1), "status": None}


def _exact_in_chunks(s, R, case):
    p = _params(case, 0)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    chunk = max(1, int(2e8 // (s.n_electrons * s.n_basis * 8)))
    parts = [_evaluate_exact(s, torch.from_numpy(R[i:i + chunk]).to(dev), p.dt, p.qf_modification != QMCB_QF_NONE)
             for i in range(0, len(R), chunk)]
    return {k: None if parts[0][k] is None else torch.cat([q[k] for q in parts]) for k in OUTPUTS}


def exact(case, seed):
    if case["kind"] not in ("evaluate", "moved", "device"):
        return None
    s = _system(case)
    if case["kind"] == "evaluate":
        return _exact_in_chunks(s, _evaluated_positions(case, seed), case)
    _, _, targets = _move_targets(case, seed)
    return [_exact_in_chunks(s, R, case) for R in targets[0]]
