"""Runs every kind of handle, ends the process's device context and runs them again: the
second run meets a device that knows nothing of the first, as another device of the process
would.  Prints one line per kind: its name and whether the two runs agree."""
import ctypes as C
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import numpy as np

import sunhubbardmy_b200 as sb
from sunhubbardmy_b200.learned import EffectiveAction

FT = dict(lattice=1, l1=8, l2=8, beta=0.4, dtau=0.1, rhub=4.0, nflr=2, kinetic=0, update=1, hs=1, nwrap=2, nublock=32)
TV = dict(lattice=2, l1=6, l2=6, beta=0.4, dtau=0.1, rv=1.0, nflr=1, kinetic=0, update=1, nwrap=2, nublock=16)
CASES = {
    "proj": dict(TV, proj=1, rndness=1e-3, update=2, rhub=0.0),
    "small": FT,
    "team": dict(FT, l1=10, l2=10),
    "fft": dict(FT, l1=16, l2=16, kinetic=1),
    "dense": dict(FT, lattice=2, l1=6, l2=6, kinetic=2),
    "bond": TV,
    "bond_direct": dict(TV, nublock=1),
    "plaquette": dict(FT, l1=10, l2=10, rhub_plq=1.0, theta=0.25),
}


def run(kind):
    if kind == "action":
        nn = EffectiveAction(8, 4, max_batch=2, seed=3)
        return nn.gradient(np.ones((2, 8, 4, 4), np.int8), np.ones(2))
    with sb.Dqmc(sb.DqmcParams.make(**CASES[kind]), n_chains=2, seeds=[sb.test_seed(0), sb.test_seed(1)]) as g:
        g.sweep_start()
        g.obser_init()
        g.sweeps(1, True)
        return g.green(1), g.bins_raw(1)


kinds = list(CASES) + ["action"]
first = {k: run(k) for k in kinds}
runtime = next(line.split()[-1] for line in open("/proc/self/maps") if "libcudart" in line)
assert C.CDLL(runtime).cudaDeviceReset() == 0
for k in kinds:
    try:
        # the network's gradient sums by atomics
        same = all(np.allclose(a, b, rtol=1e-5) if k == "action" else np.array_equal(a, b) for a, b in zip(run(k), first[k]))
    except sb.DqmcError as e:
        same = e
    print(k, same, flush=True)
