"""Sizes whose layout lies in the last bytes of a block's shared memory, where the
kernel's own variables no longer fit beside it (each kernel's largest sizes or
logs): the next kernel, or the next smaller log, runs them.  Against the oracle,
bit for bit."""
import numpy as np
import pytest

import brawl_gb300 as B
from oracle import oracle as O
from tests.test_gpu_metropolis import conc_vector, random_V
from tests.test_gpu_shared_fields import _same_stream
from tests.test_gpu_wang_landau import _emulate

pytestmark = pytest.mark.gpu


def _model(lattice, n, ns, nsh):
    V = random_V(np.random.default_rng(ns + nsh), ns, nsh)
    return V, O.OracleModel(lattice, *n, V), B.Setup(lattice, *n, ns, nsh)


@pytest.mark.parametrize("case", [
    ("bcc", (16, 16, 16), 7, 5, 1),             # fields
    ("bcc", (17, 17, 17), 6, 6, 1),
    ("fcc", (12, 12, 12), 8, 5, 1),
    ("bcc", (13, 13, 13), 10, 9, 1),            # (with a shell that lacks an opposite)
    ("simple_cubic", (30, 30, 30), 3, 1, 1),    # rounds of trials, a byte a site
    ("bcc", (47, 47, 47), 11, 4, 1),
    ("bcc", (59, 59, 59), 5, 10, 1),            # and half a byte
    ("bcc", (47, 47, 48), 6, 8, 153),           # the lattice alone
], ids=lambda c: f"{c[0]}-{c[1]}-s{c[2]}-sh{c[3]}-{c[4]}")
def test_chains_match_oracle(case):
    lattice, n, ns, nsh, chains = case
    V, mod, setup = _model(lattice, n, ns, nsh)
    beta = 1.0 / (900.0 * B.K_B_IN_RY)
    b = B.Batch([dict(setup=setup, V=V, seed=60 + c, beta=beta, species_concentrations=conc_vector(ns))
                 for c in range(chains)])
    acc = b.metropolis(400)
    for c in {0, chains - 1}:
        r = O.OracleRng(60 + c)
        cfg, _ = mod.initial_setup(r, conc_vector(ns))
        a, _ = mod.mc_run(cfg, r, beta, 400, False)
        assert acc[c] == a
        assert np.array_equal(b.config(c), cfg)
        assert _same_stream(b.rng_state(c), r)


@pytest.mark.parametrize("case", [
    ("bcc", (31, 31, 33), 12, 9),          # rounds of steps
    ("simple_cubic", (30, 30, 30), 5, 2),  # one warp's steps
], ids=lambda c: f"{c[0]}-{c[1]}-s{c[2]}-sh{c[3]}")
def test_nested_sampling_matches_oracle(case):
    lattice, n, ns, nsh = case
    V, mod, setup = _model(lattice, n, ns, nsh)
    limits, walkers, energies, _ = mod.ns_run(O.OracleRng(3), conc_vector(ns), None, 2, 150, 2)
    run = B.NestedSampling([dict(setup=setup, V=V, seed=3, n_walkers=2, n_steps=150,
                                 species_concentrations=conc_vector(ns))])
    assert np.array_equal(run.iterate(2)[0], limits)
    assert np.array_equal(run.energies(0), energies)
    for w in range(2):
        assert np.array_equal(run.walker_config(0, w), walkers[w])


@pytest.mark.parametrize("case", [
    ("bcc", (12, 12, 12), 4, 4, 5604),   # fields: a log of 64 moves, 32 and 16
    ("bcc", (12, 12, 12), 4, 4, 5919),
    ("bcc", (12, 12, 12), 4, 4, 6076),
    ("bcc", (12, 12, 12), 3, 4, 11831),  # gathered
], ids=lambda c: f"{c[0]}-{c[1]}-s{c[2]}-sh{c[3]}-{c[4]}")
def test_wang_landau_matches_oracle(case):
    lattice, n, ns, nsh, bins = case
    V, mod, setup = _model(lattice, n, ns, nsh)
    rng = O.OracleRng(8)
    cfg, _ = mod.initial_setup(rng, conc_vector(ns))
    e0 = mod.total_energy(cfg)
    edges = e0 - 4.0 + np.arange(bins + 1) * (8.0 / bins)
    walkers = [dict(setup=setup, V=V, seed=40, config=cfg.copy(), start_idx=1, end_idx=bins, window=0)]
    lngs, hists, cfgs, rngs = [np.zeros(bins)], [np.zeros(bins)], [cfg.copy()], [O.OracleRng(40)]
    wl = B.WangLandauWalkers(walkers, edges)
    acc = _emulate([mod], cfgs, rngs, walkers, edges, lngs, hists, 800, 0.05, 3)
    assert list(wl.sweeps(800, 0.05, 3)) == acc
    assert np.array_equal(wl.lng(0), lngs[0]) and np.array_equal(wl.hist(0), hists[0])
    assert np.array_equal(wl.config(0), cfgs[0])


@pytest.mark.parametrize("case", [
    ("bcc", (18, 18, 18), 4, 4),   # a log of 64 moves
    ("bcc", (17, 17, 17), 6, 4),   # of 16: gathered
], ids=lambda c: f"{c[0]}-{c[1]}-s{c[2]}-sh{c[3]}")
def test_enter_windows_matches_oracle(case):
    lattice, n, ns, nsh = case
    V, mod, setup = _model(lattice, n, ns, nsh)
    rng = O.OracleRng(70)
    cfg, _ = mod.initial_setup(rng, conc_vector(ns))
    e0 = mod.total_energy(cfg)
    edges = e0 + np.array([-900.0, -899.0, 0.0, 1.0])
    W = B.WangLandauWalkers([dict(setup=setup, V=V, seed=70, config=cfg.copy(), start_idx=1, end_idx=1, window=0)], edges)
    hi_mev = 2.0 * 13605.693122 / mod.n_atoms
    with pytest.raises(B.BrawlError):  # out of reach
        W.enter_windows(0.0, hi_mev, conc_vector(ns), None, initial=True, max_steps=600)
    f32 = np.float32
    x = float((f32(0.0025) * abs(f32(hi_mev) - f32(0.0))) * f32(mod.n_atoms)) / (13.605693122 * 1000.0)
    s = O.OracleRng(70)
    c, _ = mod.initial_setup(s, conc_vector(ns))
    mod.wl_enter_window(c, s, conc_vector(ns), None, edges[0], edges[1], 2.0 * (x * x), 600)
    assert np.array_equal(W.config(0), c)
    assert np.array_equal(W.genrand(0, 10), np.array([s.uniform() for _ in range(10)]))
