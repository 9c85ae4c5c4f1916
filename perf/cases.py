"""The work that users of this package give it, as cases that can be timed and compared.

A case is one call (or the few calls of one bin) of a program that samples with the package:

* ``sweep``: a finite-temperature run's loop body, ``obser_init``, ``sweeps`` and the read-back of the HS fields and bins,
  for one chain (the drop-in for one MPI rank) up to hundreds of batched chains, on every lattice and kinetic term;
  with ``v`` > 0 the t-V bond field is sampled, with ``ltau`` the unequal-time pass runs too;
* ``proj``: the same for the projective (ground-state) path, walkers batched;
* ``start``: new HS fields go in (``set_conf_all``), the UDV stack and G are built (``sweep_start``), G comes out;
* ``action``: the learned effective action's value and gradient on a batch of fields.

HS fields of a fresh start are drawn by the package from one seed per chain, as a fresh run draws them.
"""
import math

import numpy as np
import torch

import sunhubbardmy_b200 as sb
from sunhubbardmy_b200.learned import EffectiveAction

LATTICE = {"square": sb.SQUARE, "honeycomb": sb.HONEYCOMB, "chain": sb.CHAIN, "cubic": sb.CUBIC}
KINETIC = {"checkerboard": sb.CHECKERBOARD, "fft": sb.FFT, "dense": sb.DENSE}
UPDATE = {"fast": sb.FAST, "delay": sb.DELAY, "submatrix": sb.SUBMATRIX}
HS = {"exact": sb.EXACT, "general": sb.GENERAL4}
CHANNELS = 32                      # of the effective action's two hidden layers


def listed():
    base = {"kind": "sweep", "lattice": "square", "kinetic": "checkerboard", "update": "delay", "hs": "exact", "nflr": 2,
            "u": 4.0, "v": 0.0, "dtau": 0.1, "nwrap": 10, "nublock": 0, "sweeps": 1, "ltau": False}
    return [
        # the smallest run there is, one chain of 16 sites: launches and latency are all of it
        dict(base, name="square4-1", l="4", chains="1", update="fast", ltrot=40, sweeps=4),
        # the single-chain drop-in of the 16 x 16 lattice, half the length of its benchmark run
        dict(base, name="square16-1", l="16", chains="1", kinetic="fft", hs="general", dtau=0.05, ltrot=100, nublock=32),
        # the same lattice batched until the device is full, at a high temperature
        dict(base, name="square16-296", l="16", chains="296", kinetic="fft", hs="general", dtau=0.05, ltrot=40, nublock=32),
        # one chain of SU(4) fermions on an odd honeycomb size
        dict(base, name="honeycomb9-1", lattice="honeycomb", l="9", chains="1", update="submatrix", nflr=4, u=6.0, ltrot=40, nublock=32),
        # chains of three lattice sizes in one handle
        dict(base, name="honeycomb-mixed-128", lattice="honeycomb", l="6,9,12", chains="48,48,32", update="submatrix", nflr=4, u=6.0,
             ltrot=20, nublock=32),
        # the largest benchmarked lattice (400 sites), a few chains
        dict(base, name="square20-16", l="20", chains="16", u=6.0, ltrot=20),
        # the bond field at finite temperature
        dict(base, name="honeycomb12-tv-16", lattice="honeycomb", l="12", chains="16", nflr=1, u=0.0, v=1.0, ltrot=10, nublock=32),
        # a three-dimensional lattice, a handful of chains
        dict(base, name="cubic6-8", lattice="cubic", l="6", chains="8", hs="general", ltrot=20),
        # a run that measures unequal-time correlations as well
        dict(base, name="square8-tau-16", l="8", chains="16", kinetic="fft", hs="general", dtau=0.05, ltrot=20, ltau=True),
        # ground state: the batched walkers of the t-V model
        dict(base, name="honeycomb12-proj-64", kind="proj", lattice="honeycomb", l="12", chains="64", update="submatrix", nflr=1, u=0.0, v=1.0,
             ltrot=20, nublock=32),
        # Green's functions of many given fields, on a size that is no power of two
        {"name": "square10-start-64", "kind": "start", "l": 10, "chains": 64, "u": 4.0, "dtau": 0.1, "ltrot": 40, "nwrap": 10},
        # one minibatch of training the effective action
        {"name": "action20-16", "kind": "action", "l": 20, "ltrot": 120, "batch": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["sweep", "sweep", "sweep", "sweep", "proj", "start", "action"])
    while True:
        if kind == "action":
            case = {"kind": kind, "l": rng.randrange(4, 21), "ltrot": 4 * _log(rng, 3, 30), "batch": _log(rng, 1, 32)}
        elif kind == "start":
            case = {"kind": kind, "l": rng.randrange(4, 21), "chains": _log(rng, 1, 296), "u": rng.choice([2.0, 4.0, 6.0]), "dtau": 0.1,
                    "ltrot": rng.randrange(10, 61), "nwrap": rng.choice([5, 8, 10])}
        else:
            case = _draw_sweep(rng, kind)
        w = work(case)
        if _seconds(case) < 0.35 and w["flops"] < work(listed()[2])["flops"]:
            return case


def _draw_sweep(rng, kind):
    lattice = rng.choice(["square", "square", "honeycomb", "honeycomb", "chain", "cubic"] if kind == "sweep" else ["square", "honeycomb"])
    bond = rng.random() < (0.2 if kind == "sweep" else 0.7) and lattice == "honeycomb"
    if lattice == "square":
        l = 2 * rng.randrange(2, 11)
    elif lattice == "honeycomb":
        l = rng.randrange(3, 14)
    elif lattice == "chain":
        l = 2 * rng.randrange(4, 100)
    else:
        l = rng.choice([4, 6])
    l, chains = str(l), str(_log(rng, 1, 296))
    if kind == "sweep" and lattice == "honeycomb" and rng.random() < 0.25:
        l = "%s,%d" % (l, rng.randrange(3, 10))
        chains = "%s,%d" % (chains, _log(rng, 1, 48))
    case = {"kind": kind, "lattice": lattice, "l": l, "chains": chains,
            "kinetic": rng.choice(["checkerboard", "fft", "fft"]) if lattice == "square" else rng.choice(["checkerboard", "checkerboard", "dense"]),
            "update": rng.choice(["fast", "delay", "submatrix"]), "hs": rng.choice(["exact", "general"]),
            "nflr": 1 if bond else rng.choice([2, 2, 4]), "u": 0.0 if bond else rng.choice([2.0, 4.0, 6.0]), "v": 1.0 if bond else 0.0,
            "dtau": 0.05 if kind == "sweep" else 0.1, "nwrap": rng.choice([5, 8, 10]), "nublock": rng.choice([0, 16, 32, 64]),
            "ltrot": rng.randrange(10, 81), "sweeps": 1, "ltau": kind == "sweep" and not bond and rng.random() < 0.15}
    if bond and case["update"] == "fast":
        case["update"] = "delay"
    return case


def _ints(text):
    return [int(x) for x in str(text).split(",")]


def _sites(lattice, l):
    return {"square": l * l, "honeycomb": 2 * l * l, "chain": l, "cubic": l ** 3}[lattice]


def _sizes(case):
    """(sites, chains) of each size class."""
    if case["kind"] == "start":
        return [(case["l"] ** 2, case["chains"])]
    return [(_sites(case["lattice"], l), c) for l, c in zip(_ints(case["l"]), _ints(case["chains"]))]


def _seconds(case):
    """A rough time of a pass, to keep drawn cases no longer than listed ones: a chain's slices are one after the other."""
    if case["kind"] == "action":
        return 1e-8 * case["ltrot"] * case["l"] ** 2 * case["batch"]
    n, chains = max(s for s, _ in _sizes(case)), sum(c for _, c in _sizes(case))
    slices = case["ltrot"] * (2 * case["sweeps"] if "sweeps" in case else 1) * (2 if case.get("ltau") else 1)
    return slices * (4e-5 + 2e-3 * (n / 256) ** 2.5 * (5 if case.get("v") else 1) * max(1.0, chains / 100))


def work(case):
    """What a pass cannot do without.  Real operations of one chain of n sites: a stabilisation 56/3 n^3, a Green's function
    124/3 n^3, an accepted field change 8 n^2 (half of the proposals accepted); fields, Green's functions and bins moved once."""
    if case["kind"] == "action":
        v = case["ltrot"] * case["l"] ** 2 * case["batch"]
        layer1, layer2 = 2 * 27 * CHANNELS, 2 * 27 * CHANNELS * CHANNELS
        return {"bytes": v + 8 * (27 * CHANNELS * CHANNELS), "flops": v * (2 * layer1 + 3 * layer2)}
    flops = bytes_ = 0
    lt = case["ltrot"]
    nst = -(-lt // min(lt, case["nwrap"]))
    for n, chains in _sizes(case):
        if case["kind"] == "start":
            flops += chains * (nst * 56 / 3 * n ** 3 + 64 / 3 * n ** 3)
            bytes_ += chains * (4 * lt * n + 16 * n * n)
            continue
        s = 2 * case["sweeps"]
        if case["kind"] == "sweep":
            units = n * (3 / 2 if case["v"] else 1)
            per = nst * (56 / 3 + 124 / 3) * n ** 3 + lt * units * (8 if case["v"] else 4) * n ** 2
            per *= 2 if case["ltau"] else 1
        else:
            ne = n // 2
            units = n * (3 / 2 if case["v"] else 1)
            per = nst * (16 * (n * ne ** 2 - ne ** 3 / 3) + 17 * ne ** 3 + 24 * n * ne ** 2 + 8 * n * n * ne)
            per += lt * units * (16 if case["v"] else 8) * 2 * ne ** 2
        flops += chains * s * per
        bytes_ += chains * (8 * lt * units + 2 * 16 * n * n + 16 * 20 * n)
    return {"bytes": bytes_, "flops": flops}


def _seed(seed, c):
    return (int(seed) * 1000003 + 7919 * c + 12345) % (2 ** 31 - 1)


def _params(case, l):
    kw = dict(lattice=LATTICE[case["lattice"]], l1=l, l2=1 if case["lattice"] == "chain" else l, beta=case["dtau"] * case["ltrot"], dtau=case["dtau"],
              rhub=case["u"], rv=case["v"], nflr=case["nflr"], kinetic=KINETIC[case["kinetic"]], update=UPDATE[case["update"]], hs=HS[case["hs"]],
              nwrap=case["nwrap"], nublock=case["nublock"])
    if case["lattice"] == "cubic":
        kw["l3"] = l
    if case["kind"] == "proj":
        kw.update(proj=1, rndness=0.05)
    if case["ltau"]:
        kw.update(ltau=1, dyntau=kw["beta"])
    return sb.DqmcParams.make(**kw)


def _fields(case, seed):
    """The HS fields of a start case, one two-valued field a chain (values 1, 2)."""
    rng = np.random.default_rng(seed)
    return rng.integers(1, 3, size=(case["chains"], case["ltrot"], case["l"] ** 2), dtype=np.int32)


def _action(case, seed):
    """Weights at the scale that the network starts from, fields, and the weight of each field in the loss."""
    rng = np.random.default_rng(seed)
    parts = [(27 * CHANNELS, (3 / 27) ** 0.5), (CHANNELS, 0.1), (27 * CHANNELS * CHANNELS, (3 / (27 * CHANNELS)) ** 0.5), (CHANNELS, 0.1),
             (CHANNELS, 0.01 * (3 / CHANNELS) ** 0.5), (1, 0.01)]
    theta = np.concatenate([rng.uniform(-a, a, n) for n, a in parts]).astype(np.float32)
    fields = rng.choice(np.array([-1, 1], np.int8), size=(case["batch"], case["ltrot"], case["l"], case["l"]))
    return theta, fields, rng.standard_normal(case["batch"])


def prepare(case, seed):
    if case["kind"] == "action":
        theta, fields, r = _action(case, seed)
        net = EffectiveAction(case["ltrot"], case["l"], max_batch=case["batch"])
        net.set_params(theta)
        return {"kind": "action", "net": net, "fields": fields, "r": r}
    if case["kind"] == "start":
        p = sb.DqmcParams.make(lattice=sb.SQUARE, l1=case["l"], l2=case["l"], beta=case["dtau"] * case["ltrot"], dtau=case["dtau"], rhub=case["u"],
                               nflr=2, kinetic=sb.FFT, update=sb.DELAY, hs=sb.EXACT, nwrap=case["nwrap"])
        g = sb.Dqmc(p, n_chains=case["chains"], seeds=[_seed(seed, c) for c in range(case["chains"])])
        return {"kind": "start", "g": g, "fields": _fields(case, seed)}
    params = [p for l, n in zip(_ints(case["l"]), _ints(case["chains"])) for p in [_params(case, l)] * n]
    g = sb.Dqmc(params, n_chains=len(params), seeds=[_seed(seed, c) for c in range(len(params))])
    g.sweep_start()
    return {"kind": case["kind"], "g": g, "sweeps": case["sweeps"], "bond": case["v"] > 0, "site": case["u"] != 0, "tau": case["ltau"]}


def run(state):
    if state["kind"] == "action":
        value, grad = state["net"].gradient(state["fields"], state["r"])
        return {"value": value, "grad": grad}
    g = state["g"]
    chains = range(g.n_chains)
    if state["kind"] == "start":
        g.set_conf_all(state["fields"])
        g.sweep_start()
        return {"green": np.stack([g.green(c) for c in chains])}
    g.obser_init()
    g.sweeps(state["sweeps"], True)
    out = {"bins": np.concatenate([g.bins_raw(c) for c in chains])}
    if state["site"]:
        out["conf"] = g.conf_all()
    if state["bond"]:
        out["vconf"] = np.stack([g.vconf(c) for c in chains])
    if state["tau"]:
        out["tau"] = np.concatenate([g.dyn_bins(c).ravel() for c in chains])
    return out


def exact(case, seed):
    """A sweep's outputs follow from thousands of accept decisions in order: they have no closed value.  The start case's
    G = (1 + B)^-1 and the effective action do."""
    if case["kind"] == "action" and case["batch"] * case["ltrot"] * case["l"] ** 2 < 2_000_000:
        return _exact_action(case, seed)
    if case["kind"] == "start" and case["chains"] * (case["ltrot"] * case["l"] ** 6) < 2e11:
        return _exact_green(case, seed)
    return None


def _exact_green(case, seed):
    """G = (1 + B_lt ... B_1)^-1, B_t = K exp(V_t) K with K = exp(-dtau H0 / 2), over graded (QR) products."""
    l, n, dev = case["l"], case["l"] ** 2, "cuda" if torch.cuda.is_available() else "cpu"
    k = 2 * math.pi * torch.arange(l, dtype=torch.float64) / l
    e = (-2 * (torch.cos(k)[:, None] + torch.cos(k)[None, :])).reshape(-1)
    f = torch.exp(1j * torch.outer(k, torch.arange(l, dtype=torch.float64)))
    f = torch.kron(f, f) / l
    half = (f.conj().T @ torch.diag(torch.exp(-0.5 * case["dtau"] * e)).to(f.dtype) @ f).to(dev)
    a = math.acos(math.exp(-0.5 * case["dtau"] * case["u"]))
    diag = torch.exp(1j * a * (2.0 * torch.from_numpy(_fields(case, seed)).double().to(dev) - 3.0))
    u = torch.eye(n, dtype=half.dtype, device=dev).expand(case["chains"], n, n).contiguous()
    d = torch.ones(case["chains"], n, dtype=torch.float64, device=dev)
    v = u.clone()
    for t in range(case["ltrot"]):
        u = half @ (diag[:, t, :, None] * (half @ u))
        if (t + 1) % 4 == 0 or t + 1 == case["ltrot"]:
            u, r = torch.linalg.qr(u * d[:, None, :])
            d = torch.abs(torch.diagonal(r, dim1=1, dim2=2))
            v = (r / d[:, :, None]) @ v
    # 1 + U D V = U (U^H V^-1 + D) V, with D split into its large and small parts
    big, small = torch.clamp(d, min=1.0), torch.clamp(d, max=1.0)
    uh = u.conj().transpose(1, 2)
    m = uh / big[:, :, None] + small[:, :, None] * v
    g = torch.linalg.solve(m, uh / big[:, :, None])
    return {"green": g.cpu().numpy()}


def _exact_action(case, seed):
    theta, fields, r = _action(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p = torch.from_numpy(theta).double().to(dev).requires_grad_(True)
    parts = torch.split(p, [27 * CHANNELS, CHANNELS, 27 * CHANNELS * CHANNELS, CHANNELS, CHANNELS, 1])
    w1, b1, w2, b2, w3, b3 = parts[0].reshape(27, CHANNELS), parts[1], parts[2].reshape(27, CHANNELS, CHANNELS), parts[3], parts[4], parts[5]
    offs = [(t, y, x) for t in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]
    values = []
    for field, weight in zip(fields, r):
        s = torch.from_numpy(field).double().to(dev)
        cols = torch.stack([torch.roll(s, tuple(-o for o in off), dims=(0, 1, 2)) for off in offs], dim=-1)
        h = torch.tanh(cols @ w1 + b1)
        pre = b2 + sum(torch.roll(h, tuple(-o for o in off), dims=(0, 1, 2)) @ w2[k] for k, off in enumerate(offs))
        value = (torch.tanh(pre) @ w3).sum() + b3[0] * s.numel()
        (value * float(weight)).backward()
        values.append(float(value.detach()))
    return {"value": np.array(values), "grad": p.grad.cpu().numpy()}
