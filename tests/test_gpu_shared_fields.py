"""The kernels that keep a chain in shared memory (fields of the sites, or
gathered sums in rounds) at the edges of what they take: neighbour counts on
both sides of 64 and 128, lattices that an offset spans (a site met by two
offsets), shells without every offset's opposite, one to five fields a site,
nbr_swap, and calls of none, one and a few trials.  Against the oracle, bit for
bit: configurations, accepted moves, streams, ln g and histograms."""
import numpy as np
import pytest

import brawl_gb300 as B
from oracle import oracle as O
from tests.test_gpu_metropolis import conc_vector, random_V
from tests.test_gpu_wang_landau import _emulate

pytestmark = pytest.mark.gpu

# lattice, n, ns, nsh, nbr_swap
EDGES = [
    ("fcc", (2, 2, 2), 2, 2, False),    # offsets of n: a site is met twice
    ("bcc", (2, 3, 2), 3, 2, True),
    ("fcc", (3, 5, 7), 3, 3, True),
    ("bcc", (4, 4, 4), 5, 6, False),
    ("fcc", (4, 5, 4), 6, 6, False),    # five fields: no vector variant
    ("bcc", (5, 4, 4), 2, 10, False),   # z > 128, not every shell symmetric
    ("bcc", (4, 4, 5), 4, 8, False),
]


def _chain(case, k):
    lattice, n, ns, nsh, nbr = case
    V = random_V(np.random.default_rng(100 + k), ns, nsh)
    mod = O.OracleModel(lattice, *n, V)
    r = O.OracleRng(7000 + k)
    cfg, _ = mod.initial_setup(r, conc_vector(ns))
    return V, mod, r, cfg


@pytest.mark.parametrize("depth", [1, 2, 3, 4])
def test_chains_at_the_edges_match_oracle(depth):
    chains, ref = [], []
    for k, case in enumerate(EDGES):
        V, mod, r, cfg = _chain(case, k)
        T = (300.0, 1500.0, 6000.0)[k % 3]
        chains.append(dict(setup=B.Setup(case[0], *case[1], case[2], case[3]), V=V, seed=7000 + k,
                           beta=1.0 / (T * B.K_B_IN_RY), nbr_swap=case[4],
                           species_concentrations=conc_vector(case[2])))
        ref.append((mod, r, cfg, chains[-1]["beta"], case[4]))
    b = B.Batch(chains)
    b.set_speculation(depth)
    for trials in (0, 1, 2, 5, 64, 3001):
        acc = b.metropolis(trials)
        for k, (mod, r, cfg, beta, nbr) in enumerate(ref):
            a, _ = mod.mc_run(cfg, r, beta, trials, nbr)
            assert acc[k] == a, (EDGES[k], trials)
            assert np.array_equal(b.config(k), cfg), (EDGES[k], trials)
            assert _same_stream(b.rng_state(k), r), (EDGES[k], trials)


def _same_stream(words, r):
    g, h = O.OracleRng(1), O.OracleRng(1)
    g.set_state_words(words)
    h.set_state_words(r.state_words())
    return [g.u32() for _ in range(640)] == [h.u32() for _ in range(640)]


@pytest.mark.parametrize("wl_f,period", [(0.0, 1), (2.0 ** -31, 3), (0.05, 7), (1.5, 1), (1.0e5, 40)])
def test_wang_landau_at_the_edges_matches_oracle(wl_f, period):
    """ln f of none, below the fixed point of ln g, and beyond it."""
    for k, case in enumerate(EDGES):
        lattice, n, ns, nsh, nbr = case
        V, mod, r, cfg = _chain(case, k)
        bins = 24
        e0 = mod.total_energy(cfg)
        step = 0.004 * (1 + k % 3)
        edges = e0 - step * bins / 2 + np.arange(bins + 1) * step
        walkers, cfgs, rngs = [], [], []
        for w, (lo, hi) in enumerate([(1, bins), (9, 17), (12, 14)]):
            walkers.append(dict(setup=B.Setup(lattice, *n, ns, nsh), V=V, seed=50 + w, config=cfg.copy(),
                                start_idx=lo, end_idx=hi, window=w, nbr_swap=nbr))
            cfgs.append(cfg.copy())
            rngs.append(O.OracleRng(50 + w))
        mods = [O.OracleModel(lattice, *n, V) for _ in walkers]
        lngs = [np.zeros(bins) for _ in walkers]
        hists = [np.zeros(w["end_idx"] - w["start_idx"] + 1) for w in walkers]
        wl = B.WangLandauWalkers(walkers, edges)
        # (where a shell lacks an offset's opposite, a walk's energy is not the
        # configuration's, from which the next call starts: one call)
        for trials in (1, 2, 37, 1500) if nsh < 10 else (1500,):
            acc_o = _emulate(mods, cfgs, rngs, walkers, edges, lngs, hists, trials, wl_f, period)
            assert list(wl.sweeps(trials, wl_f, period)) == acc_o, (case, trials)
            for w in range(len(walkers)):
                assert np.array_equal(wl.lng(w), lngs[w]), (case, trials)
                assert np.array_equal(wl.hist(w), hists[w]), (case, trials)
                assert np.array_equal(wl.config(w), cfgs[w]), (case, trials)
        for w in range(len(walkers)):
            assert np.array_equal(wl.genrand(w, 20), np.array([rngs[w].uniform() for _ in range(20)]))


@pytest.mark.parametrize("scale", [1.0, 30.0])
def test_enter_windows_at_the_edges_matches_oracle(scale):
    """Walks into windows below, above and around the likely energies, one that
    is entered at the start and one that is out of reach (the configuration is
    drawn again every 250 steps a site, until max_steps), sharply biased and
    not."""
    for k, case in enumerate(EDGES):
        lattice, n, ns, nsh, _ = case
        if nsh == 10:
            continue  # (shells without every opposite: the energies never agree)
        V, mod, r, cfg = _chain(case, k)
        conc = conc_vector(ns)
        E = np.array([mod.total_energy(mod.initial_setup(O.OracleRng(s), conc)[0]) for s in range(12)])
        mid, spread = float(E.mean()), max(float(np.ptp(E)), 0.02)
        edges = mid + spread * np.array([-400.0, -399.0, -1.6, -1.0, -0.5, 0.5, 1.0, 1.6])
        walkers = [dict(setup=B.Setup(lattice, *n, ns, nsh), V=V, seed=900 + 3 * w, config=cfg.copy(), start_idx=b,
                        end_idx=b, window=w) for w, b in enumerate((1, 3, 5, 7))]
        max_steps = 250 * mod.n_atoms * 2 + 77
        lo_mev, hi_mev = 0.0, scale * spread * 13605.693122 / mod.n_atoms
        W = B.WangLandauWalkers(walkers, edges)
        try:
            W.enter_windows(lo_mev, hi_mev, conc, None, initial=True, max_steps=max_steps)
            assert False, "a window is out of reach"
        except B.BrawlError:
            pass
        f32 = np.float32
        x = float((f32(0.0025) * abs(f32(hi_mev) - f32(lo_mev))) * f32(mod.n_atoms)) / (13.605693122 * 1000.0)
        for w, d in enumerate(walkers):
            s = O.OracleRng(d["seed"])
            c, _ = mod.initial_setup(s, conc)
            mod.wl_enter_window(c, s, conc, None, edges[d["start_idx"] - 1], edges[d["end_idx"]], 2.0 * (x * x),
                                max_steps)
            assert np.array_equal(W.config(w), c), (case, w)
            assert np.array_equal(W.genrand(w, 10), np.array([s.uniform() for _ in range(10)])), (case, w)


@pytest.mark.parametrize("case", [
    ("simple_cubic", (2, 3, 4), 3, 2, False, 900),
    ("simple_cubic", (6, 5, 7), 15, 2, True, 6000),
    ("simple_cubic", (16, 3, 3), 2, 1, False, 5001),
    ("fcc", (512, 3, 40), 3, 2, False, 4000),        # half bytes; the largest coordinates
    ("bcc", (47, 47, 51), 4, 3, True, 4000),         # half bytes, a remainder of two sites
    ("fcc", (38, 38, 38), 15, 6, False, 3000),
    ("bcc", (48, 48, 50), 2, 10, False, 3000),
], ids=lambda c: f"{c[0]}-{c[1]}-s{c[2]}-sh{c[3]}")
def test_rounds_of_trials_match_oracle(case):
    """Chains in rounds of trials (simple cubic, and lattices of more than 2^16
    sites), hot and cold, in calls of none, one and many trials."""
    lattice, n, ns, nsh, nbr, trials = case
    V, mod, r, start = _chain(case[:5], ns + nsh)
    setup = B.Setup(lattice, *n, ns, nsh)
    b = B.Batch([dict(setup=setup, V=V, seed=7000 + ns + nsh, beta=1.0 / (T * B.K_B_IN_RY), nbr_swap=nbr,
                      species_concentrations=conc_vector(ns)) for T in (200.0, 4000.0)])
    cfgs, rngs = [start.copy(), start.copy()], [O.OracleRng(1), O.OracleRng(1)]
    for g in rngs:
        g.set_state_words(r.state_words())
    for k in (0, 1, 3, trials):
        acc = b.metropolis(k)
        for c, T in enumerate((200.0, 4000.0)):
            a, _ = mod.mc_run(cfgs[c], rngs[c], 1.0 / (T * B.K_B_IN_RY), k, nbr)
            assert acc[c] == a, (T, k)
            assert np.array_equal(b.config(c), cfgs[c]), (T, k)
            assert _same_stream(b.rng_state(c), rngs[c]), (T, k)


def test_rounds_of_trials_skip_a_flagged_chain():
    """A simple cubic chain whose grid holds a bad species runs no trial; the
    other one does."""
    V = random_V(np.random.default_rng(1), 3, 2)
    b = B.Batch([dict(setup=B.Setup("simple_cubic", 3, 4, 5, 3, 2), V=V, seed=9 + k, beta=100.0,
                      species_concentrations=conc_vector(3)) for k in range(2)])
    grids = b.get_configs()
    good = grids.copy()
    assert b.metropolis_host(grids, np.array([50, 60]))[1] >= 0
    bad = good.copy()
    bad[np.nonzero(bad)[0][0]] = 9
    with pytest.raises(B.BrawlError):
        b.metropolis_host(bad, np.array([50, 60]))
    cnt = b.counters()
    assert cnt[0][0] == 50 and cnt[1][0] == 120


@pytest.mark.parametrize("nsh", [2, 6])
def test_many_walkers_match_oracle(nsh):
    """More walkers than the chip has SMs, with few and with many neighbours
    (the sweeps' kernel is chosen by both)."""
    lattice, n, ns, bins = "bcc", (3, 4, 3), 3, 40
    V = random_V(np.random.default_rng(8), ns, nsh)
    mod = O.OracleModel(lattice, *n, V)
    r = O.OracleRng(5)
    walkers, cfgs, rngs = [], [], []
    E = []
    for w in range(170):
        cfg, _ = mod.initial_setup(r, conc_vector(ns))
        E.append(mod.total_energy(cfg))
        cfgs.append(cfg.copy())
        rngs.append(O.OracleRng(300 + w))
        walkers.append(dict(setup=B.Setup(lattice, *n, ns, nsh), V=V, seed=300 + w, config=cfg.copy(), start_idx=1,
                            end_idx=bins, window=w))
    span = float(np.ptp(E)) + 0.1
    edges = min(E) - span + np.arange(bins + 1) * (3 * span / bins)
    lngs = [np.zeros(bins) for _ in walkers]
    hists = [np.zeros(bins) for _ in walkers]
    wl = B.WangLandauWalkers(walkers, edges)
    assert list(wl.sweeps(250, 0.1, 5)) == _emulate([mod] * 170, cfgs, rngs, walkers, edges, lngs, hists, 250, 0.1, 5)
    for w in range(170):
        assert np.array_equal(wl.lng(w), lngs[w]) and np.array_equal(wl.hist(w), hists[w])
        assert np.array_equal(wl.config(w), cfgs[w])


@pytest.mark.parametrize("T", [300.0, 2500.0, 20000.0])
def test_many_chains_match_oracle(T):
    """More chains with fields than have their place at once: the gather kernel, in
    rounds of three, two and one trials by temperature."""
    lattice, n, ns, nsh = "bcc", (3, 3, 4), 3, 2
    V = random_V(np.random.default_rng(2), ns, nsh)
    mod = O.OracleModel(lattice, *n, V)
    beta = 1.0 / (T * B.K_B_IN_RY)
    b = B.Batch([dict(setup=B.Setup(lattice, *n, ns, nsh), V=V, seed=400 + k, beta=beta,
                      species_concentrations=conc_vector(ns)) for k in range(330)])
    acc = b.metropolis(700)
    for k in range(330):
        r = O.OracleRng(400 + k)
        cfg, _ = mod.initial_setup(r, conc_vector(ns))
        a, _ = mod.mc_run(cfg, r, beta, 700, False)
        assert acc[k] == a and np.array_equal(b.config(k), cfg), k
        if k % 40 == 0:
            assert _same_stream(b.rng_state(k), r), k


@pytest.mark.parametrize("case", [
    ("fcc", (40, 40, 40), 4, 4, False, 70),   # rounds of trials from 70 trials on
    ("bcc", (47, 47, 51), 3, 2, True, 63),    # from 63
], ids=lambda c: f"{c[0]}-{c[1]}-s{c[2]}-sh{c[3]}")
def test_calls_of_few_and_many_trials_match_oracle(case):
    """Calls on both sides of the line up to which a lattice of half bytes does not
    pay, in turn on the same chain."""
    lattice, n, ns, nsh, nbr, line = case
    V, mod, r, cfg = _chain(case[:5], ns)
    beta = 1.0 / (1200.0 * B.K_B_IN_RY)
    b = B.Batch([dict(setup=B.Setup(lattice, *n, ns, nsh), V=V, seed=7000 + ns, beta=beta, nbr_swap=nbr,
                      species_concentrations=conc_vector(ns))])
    for trials in (1, line - 1, 200, line, line + 1, 0, 2, 300):
        acc = b.metropolis(trials)
        a, _ = mod.mc_run(cfg, r, beta, trials, nbr)
        assert acc[0] == a, trials
        assert np.array_equal(b.config(0), cfg), trials
        assert _same_stream(b.rng_state(0), r), trials
