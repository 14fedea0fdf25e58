"""Records tests/golden/chains/small_spins.npz: walkers of Metropolis chains at the end of
some hundred moves.  The file was made with the library of commit e065fc0, whose
FP64 moves of small spins all ran in the one-warp-per-walker kernel k_move:

    python tests/golden/make_chains.py <that tree's root> tests/golden/chains/small_spins.npz
"""
import os
import sys

import numpy as np

# molecule, electrons (random molecules), walkers, steps, sampling, drift form, time step, refresh interval, seed.
# The first chain's walkers pass a node so closely that a rounding elsewhere
# comes back at 1e-8 of the local energies.
CHAINS = {
    "dmc_6nuc_30e": (0, 512, 600, 1, 2, 0.01, 50, 70),
    "vmc_water_10e": (0, 48, 150, 1, 2, 0.01, 20, 3),
    "vmc_water_10e plain": (0, 33, 90, 0, 0, 0.09, 0, 4),
    "random 13": (13, 40, 200, 1, 2, 0.01, 50, 5),
    "random 17": (17, 31, 200, 1, 2, 0.01, 50, 6),
    "random 10": (10, 20, 200, 1, 2, 0.01, 60, 9),
    "random 32": (32, 17, 200, 1, 2, 0.01, 60, 7),
    "random 3": (3, 16, 60, 1, 2, 0.01, 0, 8),
}
STORED = 16  # walkers whose positions are kept


def run(name):
    from qmcbeaver_b200.api import QMCB200Functions
    from qmcbeaver_b200.desc import run_params
    from qmcbeaver_b200.system import make_random_molecule, make_system
    ne, W, steps, sampling, qf, dt, refresh, seed = CHAINS[name]
    # 10 and 32 electrons have 20 nuclei, more than the walker's lanes take in one pass
    nuclei = 20 if ne in (10, 32) else max(1, ne // 5)
    s = make_random_molecule(ne, nuclei, max(4 * ne, 60 if nuclei == 20 else 0) + 1, 4.0 + ne / 10, (1, 6, 7, 8),
                             seed=ne) if ne else make_system(name.split()[0], seed=1)
    f = QMCB200Functions(s, W, run_params(sampling=sampling, qf_modification=qf, dt=dt, seed=seed,
                                          refresh_interval=refresh, rel_cutoff=0.0))
    f.init_walkers(s.initial_positions(W, seed=seed))
    f.run_steps(0, steps)
    w = f.get_walkers()
    f.close()
    return {"R": w["R"][:STORED], "e_local": w["e_local"], "log_abs_psi": w["log_abs_psi"], "sign": w["sign"]}


if __name__ == "__main__":
    out = os.path.abspath(sys.argv[2])
    os.chdir(sys.argv[1])
    sys.path.insert(0, os.getcwd())
    np.savez(out, **{f"{name}.{k}": v for name in CHAINS for k, v in run(name).items()})
