"""Paths that the number of chains of a handle selects.

* the bond field's delayed updates on teams of CTAs (a few chains of more than 64
  sites) and on one CTA per chain: fields and accept counts against the oracle;
* the equal-time measurement with eight and with two threads per bin (up to 16
  chains, more): the same chain in handles of 1 and of 17 gives the same bins.  A bin
  sums at most 64 cells of 4 slices per sweep direction in another order, so the two differ by
  less than 1e-12 of the largest bin.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TV = dict(lattice=2, l1=6, l2=6, beta=0.4, dtau=0.1, rv=1.0, nflr=1, kinetic=0, update=1, nwrap=2, nublock=16)
MEAS = {
    "square": dict(lattice=1, l1=8, l2=8, kinetic=0),
    "honeycomb": dict(lattice=2, l1=5, l2=5, kinetic=0),
    "chain": dict(lattice=3, l1=10, l2=1, kinetic=0),
    "cubic": dict(lattice=4, l1=4, l2=4, l3=4, kinetic=0),
    "r_cubic": dict(lattice=5, l1=2, l2=2, l3=2, rtd=0.7, kinetic=0),
}


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


@pytest.mark.parametrize("case", list(MEAS))
def test_measurement(sb, case):
    kw = dict(beta=0.4, dtau=0.1, rhub=3.0, nflr=2, update=1, hs=1, nwrap=2, nublock=8, **MEAS[case])
    p = sb.DqmcParams.make(**kw)
    bins = {}
    for n in (1, 17):
        with sb.Dqmc(p, n_chains=n, seeds=[sb.test_seed(c) for c in range(n)]) as g:
            g.sweep_start()
            g.obser_init()
            g.sweeps(1, True)
            bins[n] = g.bins_raw(0)
    assert np.max(np.abs(bins[1] - bins[17])) <= 1e-12 * np.max(np.abs(bins[1]))


# Chains around the 64 sites up to which a wrap is one launch: G of two half sweeps, wraps
# and B products included, against the oracle (fields equal).
PROP = {
    "square64": dict(lattice=1, l1=8, l2=8),
    "square72": dict(lattice=1, l1=6, l2=12),
    "honeycomb64": dict(lattice=2, l1=4, l2=8),
    "chain8": dict(lattice=3, l1=8, l2=1),
    "cubic64": dict(lattice=4, l1=4, l2=4, l3=4),
}


@pytest.mark.parametrize("case", list(PROP))
def test_small_chain_propagation(sb, oracle, case):
    kw = dict(beta=0.6, dtau=0.1, rhub=3.0, mu=0.2, nflr=2, kinetic=0, update=1, hs=1, nwrap=4, nublock=8, **PROP[case])
    with sb.Dqmc(sb.DqmcParams.make(**kw), n_chains=2, seeds=[sb.test_seed(c) for c in range(2)]) as g:
        g.sweep_start()
        g.sweep_b0(); g.sweep_0b()
        m = oracle.Model(**kw)
        for c in range(2):
            o = oracle.Chain(m, sb.test_seed(c))
            o.sweep_start(); o.sweep_b0(); o.sweep_0b()
            assert np.array_equal(g.conf(c), o.conf())
            assert np.max(np.abs(g.green(c) - o.green())) < 1e-10


@pytest.mark.parametrize("n", [1, 6, 40, 160])
def test_bond_updates_with_rejections(sb, oracle, n):
    """A strong coupling rejects bonds often, the family's last one among them, so flushes
    follow rejected bonds; the columns pending then range up to the 64 of a family's flush."""
    kw = dict(TV, l1=7, l2=6, rv=4.0, nwrap=1, nublock=64)
    with sb.Dqmc(sb.DqmcParams.make(**kw), n_chains=n, seeds=[sb.test_seed(c) for c in range(n)]) as g:
        g.sweep_start()
        g.sweep_b0(); g.sweep_0b()
        m = oracle.Model(**kw)
        for c in sorted({0, n - 1}):
            o = oracle.Chain(m, sb.test_seed(c))
            o.sweep_start(); o.sweep_b0(); o.sweep_0b()
            d = g.diag(c)
            assert d["accepted_v"] < 0.9 * d["proposed_v"]
            assert np.array_equal(g.vconf(c), o.vconf())
            assert d["accepted_v"] == o.diag()["accepted_v"]
            assert np.max(np.abs(g.green(c) - o.green())) < 1e-10


@pytest.mark.parametrize("case", ["square64", "honeycomb64", "cubic64", "square36", "honeycomb50", "r_cubic48", "chain62"])
def test_b_products_of_few_and_many_chains(sb, case):
    """The start-up's G of one chain comes from B products alone: in one launch or in the
    general passes, by the number of chains and sites, with the same operations on every
    element, so G of the same field has the same bits in handles of 1, 2 and 160 chains."""
    lat = {**PROP, "square36": dict(lattice=1, l1=6, l2=6), "honeycomb50": dict(lattice=2, l1=5, l2=5),
           "r_cubic48": dict(lattice=5, l1=2, l2=2, l3=2, rtd=0.7), "chain62": dict(lattice=3, l1=62, l2=1)}[case]
    kw = dict(beta=0.6, dtau=0.1, rhub=3.0, mu=0.2, nflr=2, kinetic=0, update=1, hs=1, nwrap=4, nublock=8, **lat)
    G = []
    for n in (1, 2, 160):
        with sb.Dqmc(sb.DqmcParams.make(**kw), n_chains=n, seeds=[sb.test_seed(c) for c in range(n)]) as g:
            g.sweep_start()
            G.append(g.green(0))
    assert np.array_equal(G[0], G[1]) and np.array_equal(G[0], G[2])
