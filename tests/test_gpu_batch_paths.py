"""Paths that the number of chains of a handle selects.

* the bond field's delayed updates on teams of CTAs (a few chains of more than 64
  sites) and on one CTA per chain: fields and accept counts against the oracle.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TV = dict(lattice=2, l1=6, l2=6, beta=0.4, dtau=0.1, rv=1.0, nflr=1, kinetic=0, update=1, nwrap=2, nublock=16)


@pytest.mark.parametrize("n", [1, 6, 40, 160])
def test_bond_updates(sb, oracle, n):
    with sb.Dqmc(sb.DqmcParams.make(**TV), n_chains=n, seeds=[sb.test_seed(c) for c in range(n)]) as g:
        g.sweep_start()
        g.sweep_b0(); g.sweep_0b()
        m = oracle.Model(**TV)
        for c in sorted({0, n - 1}):
            o = oracle.Chain(m, sb.test_seed(c))
            o.sweep_start(); o.sweep_b0(); o.sweep_0b()
            assert np.array_equal(g.vconf(c), o.vconf())
            assert g.diag(c)["accepted_v"] == o.diag()["accepted_v"]
            assert np.max(np.abs(g.green(c) - o.green())) < 1e-10
