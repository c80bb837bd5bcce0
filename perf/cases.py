"""The work a user of this package has it do, as cases to be timed: single
chains, batches of replicas, Wang-Landau walkers, nested sampling, set-up and
the measurements taken on configurations, each through the public classes.

A case is a dict of plain values; listed() names the ones that are followed,
draw() gives others of the same ranges.  prepare() makes what a program has in
hand before the call, run() is one pass of it, work() what a pass cannot do
without, exact() the outputs in plain 64-bit numpy where there are such.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import brawl_gb300 as B

LATTICE_SITES = {"sc": 8, "bcc": 2, "fcc": 4}
MAX_SHELLS = {"sc": 2, "bcc": 6, "fcc": 6}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # the smallest call: one sweep of the smallest chain (the serial
        # Metropolis example's lattice), its energy and its configuration
        dict(name="chain_call_fcc4", kind="call", lattice="fcc", L=4, species=5, shells=6, T=300.0, trials=256,
             nbr=False),
        # one annealing chain, the energy taken every sweep (the reference's
        # serial use: fcc 8^3, two species, two shells)
        dict(name="anneal_fcc8_binary", kind="anneal", lattice="fcc", L=8, species=2, shells=2, T=900.0, sweeps=16,
             nbr=False),
        # the headline workload: 1024 bcc replicas of four sizes from 100 K
        # to 3000 K, their configurations in page-locked host memory
        dict(name="replicas_bcc_1024", kind="replicas", lattice="bcc", sizes="8,12,16,24", chains=1024, species=4,
             shells=6, T_lo=100.0, T_hi=3000.0, sweeps=2.0, nbr=False),
        # a Monte Carlo ensemble with nearest-neighbour swaps, odd size, the
        # sampling sums on the device and the short-range order at the end
        dict(name="ensemble_fcc7_nbr", kind="ensemble", lattice="fcc", L=7, chains=48, species=3, shells=4, T=700.0,
             sweeps=8, nbr=True),
        # simple cubic replicas
        dict(name="replicas_sc_128", kind="replicas", lattice="sc", sizes="6,8", chains=128, species=3, shells=2,
             T_lo=300.0, T_hi=1500.0, sweeps=2.0, nbr=False),
        # the largest lattices: 256,000 sites, more than shared memory holds
        dict(name="replicas_fcc40_large", kind="replicas", lattice="fcc", sizes="40", chains=8, species=4, shells=4,
             T_lo=300.0, T_hi=1500.0, sweeps=0.1, nbr=False),
        # Wang-Landau: 32 windows of 4 walkers, sweeps between two replica
        # exchanges, the windows' averages
        dict(name="wang_landau_bcc12", kind="wl", lattice="bcc", L=12, windows=32, per_window=4, species=4, shells=4,
             bins=8000, trials=10000, ln_f=0.05, nbr=False),
        # Wang-Landau burn-in: every walker's biased walk into its window
        dict(name="enter_windows_bcc4", kind="enter", lattice="bcc", L=4, windows=4, per_window=8, species=4, shells=6,
             bins=512),
        # one nested-sampling run, K = 1024 walkers, 2000-step walks
        dict(name="nested_fcc6_k1024", kind="ns", lattice="fcc", L=6, runs=1, species=5, shells=3, walkers=1024,
             steps=2000, iterations=8),
        # many small nested-sampling runs side by side
        dict(name="nested_bcc5_64runs", kind="ns", lattice="bcc", L=5, runs=64, species=3, shells=4, walkers=128,
             steps=500, iterations=8),
        # measurements on given configurations: total energies and the
        # radial densities of every chain
        dict(name="measure_fcc12", kind="measure", lattice="fcc", L=12, chains=16, species=4, shells=6, wc=4),
        # set-up of a batch: chains made, their configurations drawn on the
        # device, the first energies
        dict(name="setup_bcc_256", kind="setup", lattice="bcc", sizes="8,12,16,24", chains=256, species=4, shells=6),
    ]


def _log_int(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["call", "anneal", "replicas", "replicas", "ensemble", "wl", "enter", "ns", "measure", "setup"])
    lattice = rng.choice(["fcc", "bcc"])
    species, shells = rng.randint(2, 5), rng.randint(1, 6)
    T = round(math.exp(rng.uniform(math.log(200.0), math.log(3000.0))), 1)
    nbr = rng.random() < 0.25
    if kind == "call":
        L = rng.randint(3, 10)
        return dict(kind=kind, lattice=lattice, L=L, species=species, shells=shells, T=T,
                    trials=_log_int(rng, 100, 4000), nbr=nbr)
    if kind == "anneal":
        L = rng.randint(4, 12)
        N = LATTICE_SITES[lattice] * L ** 3
        return dict(kind=kind, lattice=lattice, L=L, species=species, shells=shells, T=T,
                    sweeps=max(1, min(30, 40000 // N)), nbr=nbr)
    if kind == "replicas":
        lattice = rng.choice(["fcc", "bcc", "bcc", "sc"])
        shells = min(shells, MAX_SHELLS[lattice])
        top = {"sc": 9, "bcc": 22, "fcc": 17}[lattice]
        if lattice != "sc" and rng.random() < 0.2:  # a size that shared memory does not hold
            L = rng.randint(28, 40) if lattice == "fcc" else rng.randint(40, 48)
            return dict(kind=kind, lattice=lattice, sizes=str(L), chains=rng.randint(1, 8), species=species,
                        shells=shells, T_lo=T, T_hi=round(T * 2.0, 1), sweeps=round(rng.uniform(0.03, 0.08), 3), nbr=nbr)
        sizes = sorted({rng.randint(4, top) for _ in range(rng.randint(1, 3))})
        chains = _log_int(rng, 2, 600)
        return dict(kind=kind, lattice=lattice, sizes=",".join(map(str, sizes)), chains=chains, species=species,
                    shells=shells, T_lo=T, T_hi=round(T * rng.uniform(1.0, 3.0), 1), sweeps=1.0, nbr=nbr)
    if kind == "ensemble":
        L = rng.randint(4, 10)
        return dict(kind=kind, lattice=lattice, L=L, chains=_log_int(rng, 2, 128), species=species, shells=shells,
                    T=T, sweeps=max(1, min(12, 20000 // (LATTICE_SITES[lattice] * L ** 3))), nbr=nbr)
    if kind == "wl":
        return dict(kind=kind, lattice=lattice, L=rng.randint(4, 9 if lattice == "fcc" else 12), windows=rng.randint(1, 32),
                    per_window=rng.randint(1, 4), species=species, shells=rng.randint(1, 5), bins=_log_int(rng, 500, 8000),
                    trials=_log_int(rng, 1000, 8000), ln_f=rng.choice([1.0, 0.05, 0.001]), nbr=nbr)
    if kind == "enter":
        return dict(kind=kind, lattice=lattice, L=rng.randint(3, 5), windows=rng.randint(1, 5),
                    per_window=rng.randint(1, 4), species=species, shells=rng.randint(2, 6), bins=_log_int(rng, 128, 1024))
    if kind == "ns":
        return dict(kind=kind, lattice=lattice, L=rng.randint(4, 7), runs=_log_int(rng, 1, 96), species=species,
                    shells=rng.randint(1, 5), walkers=_log_int(rng, 32, 512), steps=_log_int(rng, 200, 2000),
                    iterations=rng.randint(2, 6))
    if kind == "measure":
        return dict(kind=kind, lattice=lattice, L=rng.randint(5, 14), chains=_log_int(rng, 1, 24), species=species,
                    shells=shells, wc=rng.randint(2, 4))
    sizes = sorted({rng.randint(4, 20) for _ in range(rng.randint(1, 4))})
    return dict(kind="setup", lattice=lattice, sizes=",".join(map(str, sizes)), chains=_log_int(rng, 4, 256),
                species=species, shells=shells)


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _interactions(rng, species, shells) -> np.ndarray:
    """Symmetric pair interactions, uniform +-50 meV per shell, in Ry."""
    V = np.zeros((species, species, shells))
    for sh in range(shells):
        a = rng.uniform(-0.05, 0.05, size=(species, species))
        V[:, :, sh] = np.triu(a) + np.triu(a, 1).T
    return V / B.RY_TO_EV


def _equal(species) -> np.ndarray:
    return np.array([0.0] + [1.0 / species] * species)


def _beta(T):
    return 1.0 / (np.asarray(T, dtype=np.float64) * B.K_B_IN_RY)


def _stream_seed(rng) -> int:
    return int(rng.integers(1, 2 ** 31))


def _sites_mask(lattice, L) -> np.ndarray:
    z, y, x = np.meshgrid(*[np.arange(2 * L)] * 3, indexing="ij")
    if lattice == "sc":
        return np.ones(x.shape, dtype=bool)
    if lattice == "fcc":
        return (x + y + z) % 2 == 0
    return (x % 2 == y % 2) & (y % 2 == z % 2)


def _random_config(rng, lattice, L, species) -> np.ndarray:
    mask = _sites_mask(lattice, L)
    n = int(mask.sum())
    s = np.arange(n) % species + 1
    rng.shuffle(s)
    cfg = np.zeros(mask.shape, dtype=np.int8)
    cfg[mask] = s
    return cfg


def _chain_list(case, rng, sizes, V, T):
    seed0 = _stream_seed(rng)
    return [dict(setup=B.Setup(case["lattice"], L, L, L, case["species"], case["shells"]), V=V, seed=seed0 + 11 * k,
                 beta=float(_beta(T[k])), nbr_swap=bool(case.get("nbr", False)),
                 species_concentrations=_equal(case["species"])) for k, L in enumerate(sizes)]


def _sizes(case) -> list[int]:
    """The batch's chain sizes: every size of the list in turn."""
    Ls = [int(v) for v in str(case["sizes"]).split(",")]
    return [Ls[k % len(Ls)] for k in range(case["chains"])]


def _ladder_energies(case, rng, V, setup, T, seed0):
    """One chain per temperature, 30 sweeps from random: (configs, energies)."""
    b = B.Batch([dict(setup=setup, V=V, seed=seed0 + 11 * k, beta=float(_beta(t)),
                      species_concentrations=_equal(case["species"])) for k, t in enumerate(T)])
    b.metropolis(30 * setup.n_atoms)
    E = b.total_energy()
    cfgs = [b.config(k) for k in range(b.n)]
    b.close()
    return cfgs, E


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    V = _interactions(rng, case["species"], case["shells"])
    st = dict(case=case, V=V)
    if kind in ("call", "anneal"):
        L = case["L"]
        setup = B.Setup(case["lattice"], L, L, L, case["species"], case["shells"])
        cfg = _random_config(rng, case["lattice"], L, case["species"])
        ch = B.Chain(setup, V)
        ch.seed(_stream_seed(rng))
        ch.set_config(cfg)
        st.update(chain=ch, beta=float(_beta(case["T"])), n=setup.n_atoms)
    elif kind == "replicas":
        sizes = _sizes(case)
        T = np.geomspace(case["T_lo"], case["T_hi"], len(sizes))
        b = B.Batch(_chain_list(case, rng, sizes, V, T))
        grids = torch.empty(b.grid_bytes, dtype=torch.int8, pin_memory=torch.cuda.is_available()).numpy()
        b.get_configs(grids)
        trials = np.array([max(1, int(s.n_atoms * case["sweeps"])) for s in b.setups], dtype=np.int64)
        st.update(batch=b, grids=grids, trials=trials)
    elif kind == "ensemble":
        b = B.Batch(_chain_list(case, rng, [case["L"]] * case["chains"], V, [case["T"]] * case["chains"]))
        st.update(batch=b, shells=b.lattice_shells(0, 3), n=b.setups[0].n_atoms)
    elif kind == "measure":
        chains = _chain_list(case, rng, [case["L"]] * case["chains"], V, [1000.0] * case["chains"])
        for ch in chains:
            ch["config"] = _random_config(rng, case["lattice"], case["L"], case["species"])
        b = B.Batch(chains)
        st.update(batch=b, shells=b.lattice_shells(0, case["wc"]))
    elif kind == "setup":
        sizes = _sizes(case)
        st.update(chains=_chain_list(case, rng, sizes, V, [1000.0] * len(sizes)))
    elif kind in ("wl", "enter"):
        L, nw, per = case["L"], case["windows"], case["per_window"]
        setup = B.Setup(case["lattice"], L, L, L, case["species"], case["shells"])
        seed0 = _stream_seed(rng)
        T = np.repeat(np.geomspace(3000.0, 700.0, nw) if nw > 1 else np.array([1500.0]), per)
        cfgs, E = _ladder_energies(case, rng, V, setup, T, seed0)
        # walkers in order of energy: the windows go up the energy axis
        order = np.argsort(E, kind="stable")
        cfgs, E = [cfgs[k] for k in order], E[order]
        # at least the spread of random configurations' energies
        z = len(_shell_vectors(case["lattice"], case["shells"]))
        span = max(float(E[-1] - E[0]), 0.002 * math.sqrt(0.5 * z * setup.n_atoms))
        lo, hi = float(E[0]) - 0.2 * span, float(E[-1]) + 0.2 * span
        bins = case["bins"]
        edges = lo + np.arange(bins + 1) * ((hi - lo) / bins)
        of = np.clip(((E - lo) / (hi - lo) * bins).astype(int) + 1, 1, bins)
        walkers = []
        cuts = [1] + [int((of[w * per - 1] + of[w * per]) // 2) for w in range(1, nw)] + [bins]
        for w in range(nw):
            own = of[w * per:(w + 1) * per]
            pad = max(8, bins // (4 * nw))
            a, e = max(1, min(cuts[w], int(own.min())) - pad), min(bins, max(cuts[w + 1], int(own.max())) + pad)
            for k in range(per):
                walkers.append(dict(setup=setup, V=V, seed=seed0 + 7 + 11 * (w * per + k), config=cfgs[w * per + k],
                                    start_idx=a, end_idx=e, window=w, nbr_swap=bool(case.get("nbr", False))))
        st.update(walkers=B.WangLandauWalkers(walkers, edges), n=setup.n_atoms, windows=nw, per=per)
        if kind == "enter":
            to_mev = B.RY_TO_EV * 1000.0 / setup.n_atoms
            st.update(e_lo=lo * to_mev, e_hi=hi * to_mev, conc=_equal(case["species"]))
    elif kind == "ns":
        L = case["L"]
        setup = B.Setup(case["lattice"], L, L, L, case["species"], case["shells"])
        seed0 = _stream_seed(rng)
        st.update(run=B.NestedSampling([dict(setup=setup, V=V, seed=seed0 + 11 * r, n_walkers=case["walkers"],
                                             n_steps=case["steps"], species_concentrations=_equal(case["species"]))
                                        for r in range(case["runs"])]))
    else:
        raise ValueError(kind)
    return st


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "call":
        ch = state["chain"]
        acc = ch.metropolis(state["beta"], case["trials"], case["nbr"])
        return dict(accepted=acc, energy=ch.total_energy(), config=ch.config())
    if kind == "anneal":
        ch = state["chain"]
        E, acc = ch.anneal_sweeps(state["beta"], case["sweeps"], state["n"], case["nbr"])
        return dict(accepted=acc, energies=E, config=ch.config())
    if kind == "replicas":
        b = state["batch"]
        acc = b.metropolis_host(state["grids"], state["trials"])
        return dict(accepted=acc, configs=state["grids"])
    if kind == "ensemble":
        b = state["batch"]
        b.sampling_reset(3)
        E, acc = b.anneal_sweeps(case["sweeps"], state["n"], accumulate=True)
        for c in range(b.n):
            b.asro_sample(c, state["shells"], rho=False)
        T = case["T"]
        per, av = b.temperature_stats(case["sweeps"], case["sweeps"] * state["n"], T, T * B.K_B_IN_RY)
        rho, rho_av = b.asro_stats(1)
        return dict(accepted=acc, energies=E, per_chain=per, average=av, rho=rho, rho_average=rho_av)
    if kind == "wl":
        w, n = state["walkers"], state["n"]
        acc = w.sweeps(case["trials"], case["ln_f"], max(1, int(0.02 * n)))
        _, partner, exchanged = w.replica_exchange()
        flat = w.flatness()
        w.average()
        firsts = range(0, w.n, state["per"])
        return dict(accepted=acc, partner=partner, exchanged=exchanged, flatness=flat, energies=w.energies(),
                    ln_g=np.concatenate([w.lng(k) for k in firsts]),
                    hist=np.concatenate([w.hist(k) for k in firsts]))
    if kind == "enter":
        w = state["walkers"]
        steps = w.enter_windows(state["e_lo"], state["e_hi"], state["conc"], initial=True)
        return dict(steps=steps, energies=w.energies(), configs=np.concatenate([w.config(k).ravel() for k in range(w.n)]))
    if kind == "ns":
        r = state["run"]
        return dict(limits=r.iterate(case["iterations"]),
                    energies=np.concatenate([r.energies(k) for k in range(case["runs"])]))
    if kind == "measure":
        b = state["batch"]
        return dict(energies=b.total_energy(),
                    rho=np.stack([b.radial_densities(c, state["shells"]) for c in range(b.n)]))
    if kind == "setup":
        b = B.Batch(state["chains"])
        out = dict(energies=b.total_energy(), configs=b.get_configs())
        b.close()
        return out
    raise ValueError(kind)


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """bytes: the state a pass has to read and to write, once each (species
    one byte a site, ln g and histograms, streams); flops: 4z FP64 adds per
    evaluated trial (two sites before and after the swap), 2 per neighbour
    term of an energy."""
    kind, lattice, sp = case["kind"], case["lattice"], case["species"]
    z = len(_shell_vectors(lattice, case["shells"]))
    differ = 1.0 - 1.0 / sp
    stream = 2 * 2500
    per_site = LATTICE_SITES[lattice]

    def chain(N, trials):
        return 2 * N + stream, 4 * z * trials * differ

    if kind == "call":
        N = per_site * case["L"] ** 3
        b, f = chain(N, case["trials"])
        return dict(bytes=b, flops=f + z * N)
    if kind == "anneal":
        N = per_site * case["L"] ** 3
        b, f = chain(N, case["sweeps"] * N)
        return dict(bytes=b, flops=f + case["sweeps"] * z * N)
    if kind == "replicas":
        tot = [chain(per_site * L ** 3, per_site * L ** 3 * case["sweeps"]) for L in _sizes(case)]
        grids = sum(8 * L ** 3 for L in _sizes(case))
        return dict(bytes=sum(b for b, _ in tot) + 2 * grids, flops=sum(f for _, f in tot))
    if kind == "ensemble":
        N = per_site * case["L"] ** 3
        b, f = chain(N, case["sweeps"] * N)
        return dict(bytes=case["chains"] * b, flops=case["chains"] * (f + case["sweeps"] * z * N))
    if kind == "wl":
        n = case["windows"] * case["per_window"]
        N = per_site * case["L"] ** 3
        b, f = chain(N, case["trials"])
        return dict(bytes=n * (b + 32 * case["bins"] / case["windows"]), flops=n * (f + z * N))
    if kind == "enter":
        n = case["windows"] * case["per_window"]
        N = per_site * case["L"] ** 3
        b, f = chain(N, 4 * N)
        return dict(bytes=n * b, flops=n * (f + 2 * z * N))
    if kind == "ns":
        N = per_site * case["L"] ** 3
        it = case["iterations"] * case["runs"]
        return dict(bytes=it * (2 * N + 8 * case["walkers"]) + case["runs"] * stream, flops=it * case["steps"] * 4 * z)
    if kind == "measure":
        N = per_site * case["L"] ** 3
        return dict(bytes=case["chains"] * N, flops=case["chains"] * N * z * 2)
    tot = sum(per_site * L ** 3 for L in _sizes(case))
    return dict(bytes=tot + 8 * sum(L ** 3 for L in _sizes(case)) + case["chains"] * stream, flops=tot * z)


# ---------------------------------------------------------------------------
# plain 64-bit results
# ---------------------------------------------------------------------------
def _shell_vectors(lattice, shells) -> list[tuple[int, int, int, int]]:
    """(dx, dy, dz, shell) on the doubled grid, shells by distance."""
    r = range(-5, 6)
    if lattice == "bcc":
        ok = [(x, y, z) for x in r for y in r for z in r if x % 2 == y % 2 == z % 2]
    elif lattice == "fcc":
        ok = [(x, y, z) for x in r for y in r for z in r if (x + y + z) % 2 == 0]
    else:
        ok = [(x, y, z) for x in r for y in r for z in r]
    d = sorted({x * x + y * y + z * z for x, y, z in ok})[1:shells + 1]
    return [(x, y, z, d.index(x * x + y * y + z * z)) for x, y, z in ok if x * x + y * y + z * z in d]


def _total_energy(cfg, V, vecs) -> float:
    e = np.zeros(cfg.shape)
    here = cfg > 0
    for dx, dy, dz, sh in vecs:
        there = np.roll(cfg, (-dz, -dy, -dx), axis=(0, 1, 2))
        e[here] += V[cfg[here] - 1, there[here] - 1, sh]
    return 0.5 * float(e.sum())


def _radial(cfg, species, wc) -> np.ndarray:
    """rho[l, j, i]: species j + 1 at the l-th distance (the first is 0) per
    site of species i + 1."""
    here = cfg > 0
    z, y, x = np.nonzero(here)
    d2 = np.unique(x * x + y * y + z * z)
    want = d2[:wc]
    rho = np.zeros((wc, species, species))
    n = np.bincount(cfg[here], minlength=species + 1)[1:].astype(np.float64)
    r = range(-5, 6)
    for dx in r:
        for dy in r:
            for dz in r:
                k = np.nonzero(want == dx * dx + dy * dy + dz * dz)[0]
                if k.size == 0:
                    continue
                there = np.roll(cfg, (-dz, -dy, -dx), axis=(0, 1, 2))
                both = here & (there > 0)
                np.add.at(rho[k[0]], (there[both] - 1, cfg[both] - 1), 1.0)
    return rho / n[None, None, :]


def _words(seed):
    g = np.random.RandomState(seed)  # mt19937, init_genrand(seed)
    while True:
        for w in g.randint(0, 2 ** 32, size=4096, dtype=np.uint64):
            yield int(w)


def _simulate(case, cfg, V, seed):
    """The case's trials one by one in plain arithmetic: (accepted, energy,
    configuration)."""
    lattice, L = case["lattice"], case["L"]
    vecs = _shell_vectors(lattice, case["shells"])
    off = np.array([v[:3] for v in vecs])
    sh = np.array([v[3] for v in vecs])
    cfg = cfg.copy()
    beta = float(_beta(case["T"]))
    words = _words(seed)
    W = 2 * L

    def below(k):
        return (next(words) * k) >> 32

    def site():
        z = below(2 * L)
        if lattice == "bcc":
            return 2 * below(L) + z % 2, 2 * below(L) + z % 2, z
        x = below(2 * L)
        return x, 2 * below(L) + (x + z) % 2, z

    def energy(s):
        n = (off + np.array(s)) % W
        return float(V[cfg[s[2], s[1], s[0]] - 1, cfg[n[:, 2], n[:, 1], n[:, 0]] - 1, sh].sum())

    acc = 0
    for _ in range(case["trials"]):
        a, b = site(), site()
        sa, sb = cfg[a[2], a[1], a[0]], cfg[b[2], b[1], b[0]]
        if sa == sb:
            acc += 1
            continue
        before = energy(a) + energy(b)
        cfg[a[2], a[1], a[0]], cfg[b[2], b[1], b[0]] = sb, sa
        change = energy(a) + energy(b) - before
        if change < 0.0 or next(words) * 2.0 ** -32 < math.exp(-beta * change):
            acc += 1
        else:
            cfg[a[2], a[1], a[0]], cfg[b[2], b[1], b[0]] = sa, sb
    return acc, _total_energy(cfg, V, vecs), cfg


def exact(case, seed):
    """Energies and radial densities of given configurations, and the short
    calls' trajectories.  A trajectory with few species and shells has moves
    whose energy change is zero but for rounding, so those have no value
    here; neither have the long ones, which would take minutes."""
    kind, lattice = case["kind"], case["lattice"]
    rng = np.random.default_rng(seed)
    V = _interactions(rng, case["species"], case["shells"])
    if kind == "call" and case["species"] >= 4 and case["shells"] >= 4 and not case["nbr"]:
        cfg = _random_config(rng, lattice, case["L"], case["species"])
        stream = _stream_seed(rng)
        # prepare() draws the configuration, then the stream's seed
        acc, E, cfg = _simulate(case, cfg, V, stream)
        return dict(accepted=acc, energy=E, config=cfg)
    if kind == "measure":
        _stream_seed(rng)
        vecs = _shell_vectors(lattice, case["shells"])
        E, rho = [], []
        for _ in range(case["chains"]):
            cfg = _random_config(rng, lattice, case["L"], case["species"])
            E.append(_total_energy(cfg, V, vecs))
            rho.append(_radial(cfg, case["species"], case["wc"]))
        return dict(energies=np.array(E), rho=np.stack(rho))
    return None
