"""Performance cases of gamdpy_b200: the work a user has the package do, through its public entry points.

Kinds of a case (``case["kind"]``):
  run      one timeblock of a Simulation (``run_timeblocks``): the steps on the device, the state and the saved
           scalars back on the host.  The state goes on from pass to pass as it does from block to block of a run.
  batch    one timeblock of a SimulationBatch of independent replicas.
  forces   Evaluator.evaluate: neighbour list, forces, energies of a configuration without time stepping.
  rdf      CalculatorRadialDistribution.update on the configuration of a Simulation.
  sq       CalculatorStructureFactor.update on the configuration of a Simulation.
  adjoint  observables of an NVE trajectory and their gradient through torch.autograd.

Systems: the Kob-Andersen 80:20 mixture at density 1.2, the single-component Lennard-Jones system, and chains of
harmonically bonded beads, each on lattice sites with random displacements and Maxwell-Boltzmann velocities.
Blocks are short enough for a trajectory to be compared before chaos separates two roundings of it.
"""
import math

import numpy as np
import torch

import gamdpy_b200 as gp
from gamdpy_b200 import adjoint

KA_SIGMA = np.array([[1.0, 0.8], [0.8, 0.88]])
KA_EPSILON = np.array([[1.0, 1.5], [1.5, 0.5]])
CUT = 2.5
BLOCKS = 256  # timeblocks a Simulation of a case is made for


def listed():
    return [
        # small mixtures are what parameter sweeps and teaching runs use: latency of a step decides
        {"name": "ka_512", "kind": "run", "system": "ka", "n": 512, "rho": 1.2, "T": 0.45, "integrator": "nvt",
         "nblist": "linked lists", "skin": 0.3, "steps": 64},
        # the default small system (FCC 8x8x8, N^2 lists)
        {"name": "lj_2048", "kind": "run", "system": "lj", "n": 2048, "rho": 0.973, "T": 0.7, "integrator": "nve",
         "nblist": "N squared", "skin": 0.5, "steps": 64},
        # a production-size glass former, odd particle number
        {"name": "ka_10007", "kind": "run", "system": "ka", "n": 10007, "rho": 1.2, "T": 0.45, "integrator": "nvt",
         "nblist": "linked lists", "skin": 0.3, "steps": 64},
        # constant pressure: virials every step, a box that changes
        {"name": "lj_npt_13500", "kind": "run", "system": "lj", "n": 13500, "rho": 0.7543, "T": 2.0,
         "integrator": "npt", "nblist": "linked lists", "skin": 0.5, "steps": 24},
        {"name": "ka_65536", "kind": "run", "system": "ka", "n": 65536, "rho": 1.2, "T": 0.45, "integrator": "nvt",
         "nblist": "linked lists", "skin": 0.3, "steps": 48},
        # the largest size of the benchmark's sweep
        {"name": "ka_1048576", "kind": "run", "system": "ka", "n": 1048576, "rho": 1.2, "T": 0.45,
         "integrator": "nvt", "nblist": "linked lists", "skin": 0.3, "steps": 32},
        # a state-point sweep of small and middle systems advanced together
        {"name": "batch_24", "kind": "batch", "replicas": 24, "n_min": 256, "n_max": 16384, "steps": 48},
        # energies and forces of given configurations: bonded chains with exclusions
        {"name": "forces_chains_100000", "kind": "forces", "system": "chains", "n": 100000, "rho": 1.0, "skin": 0.3},
        # g(r) to half the box of a small mixture, and of a large liquid to a fixed range
        {"name": "rdf_ka_5000", "kind": "rdf", "system": "ka", "n": 5000, "rho": 1.2, "bins": 500, "r_max": 0.0},
        {"name": "rdf_lj_1000188", "kind": "rdf", "system": "lj", "n": 1000188, "rho": 0.84, "bins": 1000,
         "r_max": 5.0},
        # S(q) of a large liquid
        {"name": "sq_lj_1000188", "kind": "sq", "system": "lj", "n": 1000188, "rho": 0.84, "q_max": 1.1},
        # fitting pair parameters to averages of a trajectory
        {"name": "adjoint_ka_4096", "kind": "adjoint", "n": 4096, "rho": 1.2, "T": 0.6, "steps": 50,
         "checkpoint": 50},
    ]


def _between(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["run", "run", "run", "batch", "forces", "rdf", "sq", "adjoint"])
    if kind == "run":
        system = rng.choice(["ka", "ka", "lj"])
        n = _between(rng, 400, 600000)
        integrator = rng.choice(["nvt", "nvt", "nve", "npt"]) if n <= 100000 else rng.choice(["nvt", "nve"])
        nblist = "N squared" if n <= 6000 and rng.random() < 0.5 else "linked lists"
        if system == "ka":
            rho, temp = round(rng.uniform(1.15, 1.25), 3), round(rng.uniform(0.45, 0.8), 3)
        else:
            rho, temp = round(rng.uniform(0.75, 0.973), 3), round(rng.uniform(0.7, 1.2), 3)
        if integrator == "npt":
            system, rho, temp = "lj", 0.7543, 2.0
            n = max(n, 2000)
        return {"kind": "run", "system": system, "n": n, "rho": rho, "T": temp, "integrator": integrator,
                "nblist": nblist, "skin": rng.choice([0.3, 0.4, 0.5]),
                "steps": rng.choice([18, 24]) if integrator == "npt" else rng.choice([32, 40, 48, 64])}
    if kind == "batch":
        return {"kind": "batch", "replicas": rng.randint(8, 24), "n_min": rng.choice([256, 300, 500]),
                "n_max": _between(rng, 2000, 16384), "steps": rng.choice([32, 40, 48])}
    if kind == "forces":
        system = rng.choice(["chains", "ka", "lj"])
        rho = {"chains": 1.0, "ka": 1.2, "lj": 0.84}[system]
        return {"kind": "forces", "system": system, "n": _between(rng, 1000, 200000 if system != "chains" else 100000),
                "rho": rho, "skin": rng.choice([0.3, 0.5])}
    if kind == "rdf":
        system = rng.choice(["ka", "lj"])
        near = rng.random() < 0.5
        n = _between(rng, 20000, 1000000) if near else _between(rng, 500, 12000)
        return {"kind": "rdf", "system": system, "n": n, "rho": 1.2 if system == "ka" else 0.84,
                "bins": rng.randint(100, 1000), "r_max": round(rng.uniform(3.0, 5.0), 2) if near else 0.0}
    if kind == "sq":  # 10 to 24 wavelengths along an edge
        n = _between(rng, 10000, 1000000)
        return {"kind": "sq", "system": "lj", "n": n, "rho": 0.84,
                "q_max": round(rng.uniform(10.0, 24.0 if n < 500000 else 18.6) * 2 * math.pi / (n / 0.84) ** (1 / 3), 3)}
    return {"kind": "adjoint", "n": _between(rng, 500, 4096), "rho": 1.2, "T": round(rng.uniform(0.5, 0.7), 3),
            "steps": rng.choice([30, 40, 50]), "checkpoint": rng.choice([20, 25, 50])}


# --- inputs ------------------------------------------------------------------------------------------------------
def _particles(case, seed):
    """Positions, velocities (float32), types and box length of a case's system, from the seed alone."""
    rng = np.random.default_rng(seed)
    n, rho, system = case["n"], case["rho"], case["system"]
    box = (n / rho) ** (1.0 / 3.0)
    if system == "chains":  # simple cubic, one row after the other: beads of a chain are next to each other
        m = math.ceil(n ** (1.0 / 3.0) - 1e-9)
        i = np.arange(n)
        sites = np.stack([i % m, (i // m) % m, i // (m * m)], axis=1) / m
    else:  # FCC sites, as many cells as the particles need
        m = math.ceil((n / 4) ** (1.0 / 3.0) - 1e-9)
        cells = np.arange((n + 3) // 4)
        cells = np.stack([cells // (m * m), (cells // m) % m, cells % m], axis=1)
        base = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
        sites = ((cells[:, None, :] + base[None, :, :]) / m).reshape(-1, 3)[:n]
    r = (sites - 0.5) * box + rng.uniform(-0.05, 0.05, (n, 3))
    r = (r - box * np.round(r / box)).astype(np.float32)
    v = rng.standard_normal((n, 3), dtype=np.float32) * np.float32(math.sqrt(case.get("T", 1.0)))
    v -= v.mean(axis=0, dtype=np.float64).astype(np.float32)
    t = np.zeros(n, np.int32)
    if system == "ka":
        t[rng.permutation(n)[: n // 5]] = 1
    return r, v, t, box


def _configuration(case, seed, **flags):
    r, v, t, box = _particles(case, seed)
    conf = gp.Configuration(D=3, compute_flags=flags or None)
    conf["r"] = r
    conf["v"] = v
    conf.simbox = gp.Orthorhombic(3, [box, box, box])
    conf.ptype[:] = t
    conf["m"] = 1.0
    return conf


def _potential(system, shifted_potential=False, exclusions=None):
    wrap = gp.apply_shifted_potential_cutoff if shifted_potential else gp.apply_shifted_force_cutoff
    params = [KA_SIGMA, KA_EPSILON, CUT * KA_SIGMA] if system == "ka" else [1.0, 1.0, CUT]
    return gp.PairPotential(wrap(gp.LJ_12_6_sigma_epsilon), params=params, exclusions=exclusions, max_num_nbs=300)


def _chain_bonds(n):
    """Bonds (i, i + 1) of chains of ten beads."""
    i = np.arange(n - 1)
    i = i[i % 10 != 9]
    return np.stack([i, i + 1, np.zeros_like(i)], axis=1)


def _plan(conf, **values):
    return {**gp.get_default_compute_plan(conf), **values}


def _simulation(case, seed):
    flags = {"Vol": True} if case["integrator"] == "npt" else {}
    conf = _configuration(case, seed, **flags)
    dt = 0.004 if case["system"] == "lj" else 0.005
    if case["integrator"] == "nvt":
        integrator = gp.integrators.NVT(temperature=case["T"], tau=0.2, dt=dt)
    elif case["integrator"] == "npt":
        integrator = gp.integrators.NPT_Atomic(temperature=case["T"], tau=0.4, pressure=4.7, tau_p=20.0, dt=dt)
    else:
        integrator = gp.integrators.NVE(dt=dt)
    return gp.Simulation(conf, _potential(case["system"], case["integrator"] == "npt"), integrator,
                         [gp.ScalarSaver(16), gp.MomentumReset(100)], num_timeblocks=BLOCKS,
                         steps_per_timeblock=case["steps"], storage="memory",
                         compute_plan=_plan(conf, nblist=case["nblist"], skin=case["skin"]))


def _replicas(case, seed):
    """The state points of a batch: sizes spread over their logarithm, densities and temperatures uniform."""
    rng = np.random.default_rng(seed + 1000003)
    k = case["replicas"]
    n = np.exp(np.linspace(math.log(case["n_min"]), math.log(case["n_max"]), k))
    return [{"kind": "run", "system": "ka", "n": int(n[i]), "rho": float(rng.uniform(1.1, 1.3)),
             "T": float(rng.uniform(0.4, 1.0)), "integrator": "nvt", "nblist": "linked lists", "skin": 0.3,
             "steps": case["steps"]} for i in range(k)]


def _theta(eps_ab, sig_ab):
    sig, eps = KA_SIGMA.copy(), KA_EPSILON.copy()
    sig[0, 1] = sig[1, 0] = sig_ab
    eps[0, 1] = eps[1, 0] = eps_ab
    return adjoint.theta_from_tables(sig, eps)


RDF = {"bins": 40, "r_lo": 0.7, "r_hi": 2.7, "width": 0.05, "every": 10}


def _weights(seed, count):
    """Weights of a linear loss on the observables of an adjoint case."""
    return torch.as_tensor(np.random.default_rng(seed + 7).uniform(0.5, 1.5, count))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        sim = _simulation(case, seed)
        return {"kind": kind, "sim": sim, "blocks": None}
    if kind == "batch":
        sims = [_simulation(c, seed + 17 * i) for i, c in enumerate(_replicas(case, seed))]
        return {"kind": kind, "batch": gp.SimulationBatch(sims), "blocks": None}
    if kind == "forces":
        conf = _configuration(case, seed, lapU=True)
        interactions = []
        exclusions = None
        if case["system"] == "chains":
            bonds = gp.Bonds(gp.harmonic_bond_function, [[1.0, 3000.0]], _chain_bonds(case["n"]))
            exclusions = bonds.get_exclusions(conf, 2)
            interactions.append(bonds)
        interactions.insert(0, _potential(case["system"], exclusions=exclusions))
        return {"kind": kind, "conf": conf,
                "evaluator": gp.Evaluator(conf, interactions,
                                          compute_plan=_plan(conf, nblist="linked lists", skin=case["skin"]))}
    if kind in ("rdf", "sq"):
        conf = _configuration(case, seed)
        sim = gp.Simulation(conf, _potential(case["system"]), gp.integrators.NVE(dt=0.004), [], num_timeblocks=1,
                            steps_per_timeblock=16, storage="memory",
                            compute_plan=_plan(conf, nblist="linked lists", skin=0.5))
        conf.copy_to_device()
        if kind == "rdf":
            calc = gp.CalculatorRadialDistribution(conf, case["bins"], r_max=case["r_max"] or None)
        else:
            calc = gp.CalculatorStructureFactor(conf)
            calc.generate_q_vectors(case["q_max"])
        return {"kind": kind, "sim": sim, "calc": calc}
    conf = _configuration({**case, "system": "ka"}, seed)
    engine = adjoint.AdjointNVE(conf, CUT * KA_SIGMA, dt=0.005, steps=case["steps"],
                                checkpoint_every=case["checkpoint"], rdf=RDF)
    return {"kind": kind, "engine": engine, "theta": torch.tensor(_theta(1.5, 0.8)),
            "weights": _weights(seed, engine.n_obs)}


# --- one pass ------------------------------------------------------------------------------------------------------
def _next_block(state, simulation):
    """The next timeblock of a run; a new run_timeblocks when the last one has had all its blocks."""
    if state["blocks"] is not None:
        for block in state["blocks"]:
            return block
    state["blocks"] = simulation.run_timeblocks()
    return next(state["blocks"])


def _unwrapped(conf):
    """Positions without the periodic wrap, as mean-square displacements take them."""
    lengths = torch.from_numpy(np.asarray(conf.simbox.lengths, np.float32))
    return torch.addcmul(torch.from_numpy(conf["r"]), torch.from_numpy(conf.r_im).float(), lengths)


def run(state):
    kind = state["kind"]
    if kind == "run":
        sim = state["sim"]
        block = _next_block(state, sim)
        conf = sim.configuration
        return {"r": _unwrapped(conf), "v": conf["v"], "f": conf["f"], "scalars": sim.output["scalars"][block]}
    if kind == "batch":
        sims = state["batch"].simulations
        block = _next_block(state, state["batch"])
        return {"r": torch.cat([_unwrapped(s.configuration) for s in sims]),
                "v": np.concatenate([s.configuration["v"] for s in sims]),
                "f": np.concatenate([s.configuration["f"] for s in sims]),
                "scalars": np.concatenate([s.output["scalars"][block] for s in sims])}
    if kind == "forces":
        state["evaluator"].evaluate()
        conf = state["conf"]
        return {k: conf[k] for k in ("f", "U", "W", "lapU")}
    if kind == "rdf":
        state["calc"].update()
        return state["calc"].rdf_list[-1]
    if kind == "sq":
        state["calc"].update()
        return state["calc"].list_of_rho_q[-1]
    theta = state["theta"].clone().requires_grad_(True)
    obs = state["engine"].observables(theta)
    (obs * state["weights"]).sum().backward()
    return {"observables": obs.detach(), "gradient": theta.grad}


# --- what a pass cannot do without ------------------------------------------------------------------------------
def _pair_flops(system, n, rho):
    """Pairs inside the cutoff, each once, at 30 operations."""
    cut3 = CUT ** 3 * (0.64 + 0.32 * 0.512 + 0.04 * 0.88 ** 3 if system == "ka" else 1.0)
    return n * 0.5 * (4.0 / 3.0) * math.pi * cut3 * rho * 30.0


def _run_work(case):
    n, steps = case["n"], case["steps"]
    # a step reads and writes r and v; the block's end leaves r, v, f and images on the host
    return {"bytes": n * (steps * 56.0 + 48.0), "flops": steps * _pair_flops(case["system"], n, case["rho"])}


def work(case):
    kind = case["kind"]
    if kind == "run":
        return _run_work(case)
    if kind == "batch":
        parts = [_run_work(c) for c in _replicas(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, rho = case["n"], case["rho"]
    if kind == "forces":
        return {"bytes": n * 56.0, "flops": _pair_flops(case["system"], n, rho)}
    if kind == "rdf":
        box = (n / rho) ** (1.0 / 3.0)
        reach = case["r_max"] or box / 2
        return {"bytes": n * 16.0 + 8.0 * case["bins"], "flops": n * 0.5 * (4.0 / 3.0) * math.pi * reach ** 3 * rho * 10}
    if kind == "sq":
        q = math.pi / 6.0 * (case["q_max"] * (n / rho) ** (1.0 / 3.0) / (2.0 * math.pi)) ** 3
        return {"bytes": n * 16.0 + q * 28.0, "flops": n * q * 8.0}
    pairs = _pair_flops("ka", n, rho) / 30.0
    # forward once, backward with the states kept or computed again: the forces and their derivatives once each
    return {"bytes": case["steps"] * n * 112.0, "flops": case["steps"] * pairs * 150.0}


# --- the same in 64 bits -----------------------------------------------------------------------------------------
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _pairs(r, box, reach):
    """Index pairs (each once) closer than `reach` by the minimum image, r in [-box/2, box/2]."""
    n, dev = r.shape[0], r.device
    nc = int(box / reach)
    if nc < 3:
        found = []
        for lo in range(0, n, 2048):
            hi = min(n, lo + 2048)
            d = r[None, :, :] - r[lo:hi, None, :]
            d -= box * torch.round(d / box)
            i, j = torch.nonzero((d * d).sum(-1) < reach * reach, as_tuple=True)
            keep = i + lo < j
            found.append(torch.stack([i[keep] + lo, j[keep]]))
        return torch.cat(found, 1)
    c = torch.remainder(torch.floor((r / box + 0.5) * nc).long(), nc)
    cell = (c[:, 0] * nc + c[:, 1]) * nc + c[:, 2]
    order = torch.argsort(cell)
    count = torch.bincount(cell, minlength=nc ** 3)
    start = torch.cumsum(count, 0) - count
    most = int(count.max())
    table = torch.full((nc ** 3, most), -1, dtype=torch.long, device=dev)
    table[cell[order], torch.arange(n, device=dev) - start[cell[order]]] = order
    grid = torch.arange(nc ** 3, device=dev).reshape(nc, nc, nc)
    at_once = max(1, int(2e7) // (most * most))
    found = []
    for s in range(13, 27):
        other = torch.roll(grid, (1 - s // 9, 1 - (s // 3) % 3, 1 - s % 3), (0, 1, 2)).reshape(-1)
        for lo in range(0, nc ** 3, at_once):
            a, b = table[lo:lo + at_once], table[other[lo:lo + at_once]]
            d = r[b.clamp(min=0)][:, None, :, :] - r[a.clamp(min=0)][:, :, None, :]
            d -= box * torch.round(d / box)
            ok = ((d * d).sum(-1) < reach * reach) & (a >= 0)[:, :, None] & (b >= 0)[:, None, :]
            if s == 13:
                ok &= a[:, :, None] < b[:, None, :]
            k, x, y = torch.nonzero(ok, as_tuple=True)
            found.append(torch.stack([a[k, x], b[k, y]]))
    return torch.cat(found, 1)


def _tables(system, dev):
    sig, eps = (KA_SIGMA, KA_EPSILON) if system == "ka" else (np.ones((1, 1)), np.ones((1, 1)))
    single = [torch.as_tensor(x.astype(np.float32).astype(np.float64), device=dev) for x in (sig, eps)]
    return single[0], single[1], torch.as_tensor((CUT * sig).astype(np.float32).astype(np.float64), device=dev)


def _pair_terms(d, sig, eps, cut):
    """Shifted-force u(r), s = -u'(r)/r and r^2 of pairs with displacement d (zero outside the cutoff)."""
    r2 = (d * d).sum(-1)
    r = torch.sqrt(r2)
    sr6, src6 = (sig * sig / r2) ** 3, (sig / cut) ** 6
    s_cut = eps * (48 * src6 * src6 - 24 * src6) / (cut * cut)
    inside = r < cut
    s = eps * (48 * sr6 * sr6 - 24 * sr6) / r2 - s_cut
    u = 4 * eps * (sr6 * sr6 - sr6) - 4 * eps * (src6 * src6 - src6) + s_cut * cut * (r - cut)
    zero = torch.zeros_like(s)
    return torch.where(inside, u, zero), torch.where(inside, s, zero), r2, sr6, inside


def _forces(r, types, box, pairs, tables, energies=False):
    sig, eps, cut = tables
    f = torch.zeros_like(r)
    extra = [torch.zeros(r.shape[0], dtype=r.dtype, device=r.device) for _ in range(3)] if energies else None
    for lo in range(0, pairs.shape[1], 1 << 24):
        i, j = pairs[0, lo:lo + (1 << 24)], pairs[1, lo:lo + (1 << 24)]
        d = r[i] - r[j]
        d -= box * torch.round(d / box)
        ti, tj = types[i], types[j]
        u, s, r2, sr6, inside = _pair_terms(d, sig[ti, tj], eps[ti, tj], cut[ti, tj])
        fd = s[:, None] * d
        f.index_add_(0, i, fd)
        f.index_add_(0, j, -fd)
        if energies:
            second = torch.where(inside, eps[ti, tj] * (624 * sr6 * sr6 - 168 * sr6) / r2, torch.zeros_like(s))
            for acc, x in zip(extra, (0.5 * u, r2 * s / 6.0, second - 2.0 * s)):
                acc.index_add_(0, i, x)
                acc.index_add_(0, j, x)
    return (f, *extra) if energies else f


def _exact_run(case, seed):
    """Unwrapped positions, velocities and final forces of the first block, leap-frog NVE or Nose-Hoover NVT."""
    dev = _device()
    r32, v32, t, box = _particles(case, seed)
    box = float(np.float32(box))
    types = torch.as_tensor(t.astype(np.int64), device=dev)
    dt = float(np.float32(0.004 if case["system"] == "lj" else 0.005))
    tables = _tables(case["system"], dev)
    n = len(t)
    nvt, dof, omega2 = case["integrator"] == "nvt", 3 * n - 3, 4.0 * math.pi ** 2 / 0.2 ** 2
    xi, skin = 0.0, 0.6

    def start():
        return (torch.as_tensor(r32.astype(np.float64), device=dev), torch.as_tensor(v32.astype(np.float64), device=dev))

    def wrapped(r):
        return r - box * torch.round(r / box)

    r, v = start()
    pairs, at = _pairs(wrapped(r), box, CUT + skin), r.clone()
    for step in range(-1 if nvt else 0, case["steps"]):  # the constructor's test step leaves its thermostat state
        if step == 0:
            r, v = start()
        if float((r - at).abs().max()) > skin / 4:
            pairs, at = _pairs(wrapped(r), box, CUT + skin), r.clone()
        f = _forces(r, types, box, pairs, tables)
        if nvt:
            x = 0.5 * xi * dt
            v = ((1.0 - x) * v + f * dt) / (1.0 + x)
            xi += dt * omega2 * (float((v * v).sum()) / (dof * case["T"]) - 1.0)
        else:
            v = v + f * dt
        r = r + v * dt
    if float((r - at).abs().max()) > skin / 4:
        pairs = _pairs(wrapped(r), box, CUT + skin)
    return {"r": r, "v": v, "f": _forces(r, types, box, pairs, tables), "scalars": None}


def _exact_forces(case, seed):
    dev = _device()
    r32, _, t, box = _particles(case, seed)
    box = float(np.float32(box))
    r = torch.as_tensor(r32.astype(np.float64), device=dev)
    types = torch.as_tensor(t.astype(np.int64), device=dev)
    pairs = _pairs(r, box, CUT + 0.01)
    bonds = None
    if case["system"] == "chains":
        bonds = torch.as_tensor(_chain_bonds(case["n"])[:, :2].T, device=dev)
        low = torch.minimum(pairs[0], pairs[1])
        adjacent = ((pairs[0] - pairs[1]).abs() == 1) & (low % 10 != 9)
        pairs = pairs[:, ~adjacent]
    f, u, w, lap = _forces(r, types, box, pairs, _tables(case["system"], dev), energies=True)
    if bonds is not None:
        i, j = bonds
        d = r[i] - r[j]
        d -= box * torch.round(d / box)
        length = d.norm(dim=1)
        s = -3000.0 * (length - 1.0) / length
        f.index_add_(0, i, s[:, None] * d)
        f.index_add_(0, j, -s[:, None] * d)
        for k in (i, j):
            u.index_add_(0, k, 0.25 * 3000.0 * (length - 1.0) ** 2)
            w.index_add_(0, k, length * length * s / 6.0)
            lap.index_add_(0, k, 3000.0 - 2.0 * s)
    return {"f": f, "U": u, "W": w, "lapU": lap}


def _exact_sq(case, seed):
    dev = _device()
    r32, _, _, box = _particles(case, seed)
    box = float(np.float32(box))
    r = torch.as_tensor(r32.astype(np.float64), device=dev)
    n_max = int(np.ceil(case["q_max"] * box / (2 * np.pi)))
    nv = np.stack(np.meshgrid(*[np.arange(n_max)] * 3, indexing="ij"), axis=-1).reshape(-1, 3)[1:]
    nv = nv[np.linalg.norm(np.array(2 * np.pi * nv / np.float32(box), np.float32), axis=1) < case["q_max"]]
    nv = torch.as_tensor(nv, device=dev)
    acc = torch.zeros(len(nv), dtype=torch.complex128, device=dev)
    k = torch.arange(n_max, device=dev, dtype=torch.float64)
    for lo in range(0, len(r), 1 << 15):
        phase = 2 * math.pi / box * r[lo:lo + (1 << 15), :, None] * k
        e = torch.polar(torch.ones_like(phase), phase)
        xy = torch.einsum("pa,pb->pab", e[:, 0], e[:, 1]).reshape(len(e), -1)
        full = (xy.T @ e[:, 2]).reshape(n_max, n_max, n_max)
        acc += full[nv[:, 0], nv[:, 1], nv[:, 2]]
    return acc / math.sqrt(len(r))


def _exact_adjoint(case, seed):
    """Observables and their gradient through torch.autograd, in 64 bits over the pairs within reach."""
    dev = _device()
    r32, v32, t, box = _particles({**case, "system": "ka"}, seed)
    box = float(np.float32(box))
    r, v = (torch.as_tensor(x.astype(np.float64), device=dev) for x in (r32, v32))
    types = torch.as_tensor(t.astype(np.int64), device=dev)
    theta = torch.tensor(_theta(1.5, 0.8), device=dev, requires_grad=True)
    kind = torch.tensor([[0, 1], [1, 2]], device=dev)
    cut = torch.as_tensor(CUT * KA_SIGMA, device=dev)
    n, dt, width = len(t), float(np.float32(0.005)), float(np.float32(RDF["width"]))
    lo, hi, bins = float(np.float32(RDF["r_lo"])), float(np.float32(RDF["r_hi"])), RDF["bins"]
    dr = (hi - lo) / bins
    centres = lo + (torch.arange(bins, device=dev, dtype=torch.float64) + 0.5) * dr
    sums, g, samples, skin = [0.0, 0.0, 0.0], 0.0, 0, 0.6
    reach = max(CUT, RDF["r_hi"] + 8 * RDF["width"]) + skin
    at = None
    for step in range(case["steps"]):
        with torch.no_grad():
            if at is None or float((r - at).abs().max()) > skin / 4:
                at = r.detach().clone()
                pairs = _pairs(at - box * torch.round(at / box), box, reach)
        i, j = pairs
        d = r[i] - r[j]
        d = d - box * torch.round(d.detach() / box)
        k = kind[types[i], types[j]]
        u, s, r2, _, _ = _pair_terms(d, theta[3 + k], theta[k], cut[types[i], types[j]])
        fd = s[:, None] * d
        f = torch.zeros_like(r).index_add(0, i, fd).index_add(0, j, -fd)
        v_new = v + f * dt
        mean = 0.5 * (v + v_new)
        for q, x in enumerate((u.sum(), (r2 * s).sum() / 3.0, 0.5 * (mean * mean).sum())):
            sums[q] = sums[q] + x / case["steps"]
        if step % RDF["every"] == 0:
            length = torch.sqrt(r2[(types[i] == 0) & (types[j] == 0)])
            length = length[length < hi + 8 * width]
            x = length[:, None] - centres
            g = g + 2.0 * (torch.exp(-x * x / (2 * width * width)) / (math.sqrt(2 * math.pi) * width)).sum(0)
            samples += 1
        r, v = r + v_new * dt, v_new
    na = float((t == 0).sum())
    g = g / (samples * na * (na / box ** 3) * 4 * math.pi * centres * centres)
    obs = torch.cat([torch.stack(sums), g])
    (obs * _weights(seed, len(obs)).to(dev)).sum().backward()
    return {"observables": obs.detach(), "gradient": theta.grad}


def exact(case, seed):
    kind = case["kind"]
    if kind == "run":
        return _exact_run(case, seed) if case["integrator"] in ("nve", "nvt") else None
    if kind == "batch":
        parts = [_exact_run(c, seed + 17 * i) for i, c in enumerate(_replicas(case, seed))]
        return {**{k: torch.cat([p[k] for p in parts]) for k in ("r", "v", "f")}, "scalars": None}
    if kind == "forces":
        return _exact_forces(case, seed)
    if kind == "sq":
        return _exact_sq(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    return None  # counts
