"""Teams of CTAs (thread-block clusters) on one chain: the number of chains of a
handle sets the team size (16 CTAs per chain for a few chains, one per chain for
hundreds), and the chains' sizes set how columns and tiles are dealt out over a
team.  Handles of mixed sizes at every team size: the QR against its defining
properties (the bounds of test_qr_householder), start-up and one sweep against
the oracle (fields and accept counts exactly, G to 1e-10)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one column chunk of a team and its remainders: below 16, past 16, 64 and 128 columns
LENGTHS = (8, 34, 66, 98, 130)
CHAINS = (1, 6, 14, 40, 160)


def params(l):
    return dict(lattice=3, l1=l, l2=1, beta=1.2, dtau=0.1, rhub=3.0, nflr=2, kinetic=0, update=1, hs=1, nwrap=5,
                nublock=16)


def handle(sb, n):
    ps = [sb.DqmcParams.make(**params(l)) for l in (LENGTHS if n > 1 else LENGTHS[-1:])]
    return sb.Dqmc([ps[c % len(ps)] for c in range(n)], n_chains=n, seeds=[sb.test_seed(c) for c in range(n)])


@pytest.mark.parametrize("n", CHAINS)
def test_qr(sb, n):
    with handle(sb, n) as g:
        rng = np.random.default_rng(n)
        As = []
        for c in range(min(n, 5)):
            N = g.ndim(c)
            A = (rng.standard_normal((N, N)) + 1j * rng.standard_normal((N, N))) * np.logspace(8, -8, N)[None, :]
            g.set_work(0, A, c)
            As.append(A)
        ld = g.test_qr(0, 1)
        for c, A in enumerate(As):
            Q, R = g.work(1, c), np.triu(g.work(0, c))
            assert np.max(np.abs(Q.conj().T @ Q - np.eye(len(A)))) < 1e-12
            assert np.max(np.abs(Q @ R - A) / np.max(np.abs(A), axis=0)[None, :]) < 1e-12
            sign, _ = np.linalg.slogdet(Q)
            assert abs(np.exp(1j * ld[c].imag) - sign) < 1e-10 and abs(ld[c].real) < 1e-10


@pytest.mark.parametrize("n", CHAINS)
def test_sweep(sb, oracle, n):
    with handle(sb, n) as g:
        g.sweep_start()
        chains = range(min(n, 5))
        ch = []
        for c in chains:
            m = oracle.Model(**params(g.ndim(c)))
            o = oracle.Chain(m, sb.test_seed(c))
            o.sweep_start()
            assert np.max(np.abs(g.green(c) - o.green())) < 1e-10
            ch.append((m, o))
        g.sweep_b0(); g.sweep_0b()
        for c, (m, o) in zip(chains, ch):
            o.sweep_b0(); o.sweep_0b()
            assert np.array_equal(g.conf(c), o.conf())
            assert g.diag(c)["accepted"] == o.diag()["accepted"]
            assert np.max(np.abs(g.green(c) - o.green())) < 1e-10


@pytest.mark.parametrize("l, n", [(10, 1), (10, 2), (12, 9), (10, 160)])
def test_forced_flips(sb, l, n):
    """Block moves of more than 64 sites: most windows of a forced slice hold no
    forced site, so a slice's flush follows windows that accept nothing.  Local updates off,
    so the change of the log weight is the sum of the accepted blocks' log ratios
    (the bounds of test_block_moves_are_exact)."""
    from sunhubbardmy_b200.learned import EffectiveAction
    p = sb.DqmcParams.make(lattice=1, l1=l, l2=l, beta=2.0, dtau=0.1, rhub=1.0, nflr=2, kinetic=0, update=1, hs=0,
                           nwrap=10, nublock=32)
    nn = EffectiveAction(p.ltrot, l, max_batch=2 * n)
    nn.set_params(np.zeros(nn.nparams, np.float32))
    with sb.Dqmc(p, n_chains=n, seeds=[sb.test_seed(c) for c in range(n)]) as g:
        g.sweep_start()
        w0 = np.array([g.diag(c)["logweight"].real for c in range(n)])
        g.reset_diag()
        g.sweeps_learned(nn, 20, lmeasure=False, seed=77, lupdate=False)
        for c in range(n):
            d = g.diag(c)
            assert d["blk_proposed"] == d["blk_stage1"] > 0
            assert d["max_wrap_error"] < 1e-8
            w1 = d["logweight"].real
            assert abs(p.nflr * (w1 - w0[c]) - d["blk_sum_logratio"]) < 1e-7 * max(1.0, abs(w1))
        assert sum(g.diag(c)["blk_accepted"] for c in range(n)) > 0


# sites of a chain and chains of each handle
GROUPS = {"16x4": [(100, 4)] * 16, "4x20": [(130, 20)] * 4, "2x74": [(98, 74)] * 2, "3x74": [(98, 74)] * 3, "sizes": [(72, 12), (162, 8), (36, 12)],
          "2x1": [(130, 1)] * 2}


@pytest.mark.parametrize("name", list(GROUPS))
def test_concurrent_handles_share_the_device(sb, name):
    """Handles that run at once take two CTAs per SM together, and a handle by itself
    its own team again; the chains evolve exactly as in separate runs."""
    import torch
    slots = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    runs = []
    for concurrent in (True, False):
        hs = [sb.Dqmc(sb.DqmcParams.make(**params(l)), n_chains=n, seeds=[sb.test_seed(100 * k + c) for c in range(n)])
              for k, (l, n) in enumerate(GROUPS[name])]
        if concurrent:
            sb.sweep_start_concurrent(hs)
            for g in hs:
                g.obser_init()
            sb.sweeps_concurrent(hs, 2, True)
        else:
            for g in hs:
                g.sweep_start(); g.obser_init()
                g.sweeps(2, True)
        runs.append(hs)
    a, b = runs
    shared = [g.sweep_team(True) for g in a]
    assert all(t >= 1 and t <= g.sweep_team() for t, g in zip(shared, b))
    assert sum(t * g.n_chains for t, g in zip(shared, a)) <= max(slots, sum(g.n_chains for g in a))
    for ga, gb in zip(a, b):
        for c in {0, ga.n_chains - 1}:
            assert np.array_equal(ga.conf(c), gb.conf(c))
            assert np.array_equal(ga.green(c), gb.green(c))
            assert np.array_equal(ga.bins_raw(c), gb.bins_raw(c))
    a[0].sweeps(1, True)
    assert a[0].sweep_team() == b[0].sweep_team()
    for g in a + b:
        g.close()


@pytest.mark.parametrize("n", [40, 160])
@pytest.mark.parametrize("concurrent", [False, True])
def test_the_flush_depth_is_timed_with_the_teams_of_the_run(sb, monkeypatch, n, concurrent):
    """The autotuner times a few chains with the CTAs per chain that the run has."""
    from sunhubbardmy_b200 import autotune
    timed = []

    class Timed(sb.Dqmc):
        def __exit__(self, *a):
            timed.append(self.sweep_team())
            return super().__exit__(*a)

    monkeypatch.setattr(autotune, "Dqmc", Timed)
    build = autotune.size_classes if concurrent else autotune.batched
    g, _ = build([(sb.DqmcParams.make(**params(98)), n)], candidates=(16, 32))
    with g:
        g.sweep_start()
        g.sweeps(1, True)
        real = {h.sweep_team(True) for h in g.handles} if concurrent else {g.sweep_team()}
    assert set(timed[:2]) == real


def test_set_team(sb):
    """Chains of a handle with set teams: the bits of every team above one CTA are the same."""
    out = []
    for team in (2, 8, 16):
        with sb.Dqmc(sb.DqmcParams.make(**params(130)), n_chains=2, seeds=[sb.test_seed(c) for c in range(2)]) as g:
            g.set_team(team, True)
            g.sweep_start(); g.obser_init()
            g.sweeps(2, True)
            assert g.sweep_team() == team
            out.append((g.conf(1), g.green(1), g.bins_raw(1)))
            with pytest.raises(sb.DqmcError):
                g.set_team(3, True)
            with pytest.raises(sb.DqmcError):
                g.set_team(4, False)
    for a in out[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(a, out[0]))
