"""Nested-sampling walks in rounds of steps at the edges of what a round takes:
fewer steps than a round, one walker, neighbour counts in every variant, more
than seven species, one atom of a species (site 2 is redrawn for a long time),
tiny lattices where most of a round's steps share sites, and enough iterations
that the walks go from accepting everything to rejecting nearly everything.
Against the oracle, bit for bit."""
import numpy as np
import pytest

import brawl_gb300 as B
from oracle import oracle as O
from tests.test_gpu_metropolis import conc_vector, equi_numbers, random_V

pytestmark = pytest.mark.gpu

CASES = [
    # lattice, n, ns, nsh, K, n_steps, n_iter, atoms of species 1 (None: equal)
    ("fcc", (3, 3, 3), 2, 1, 8, 7, 200, None),
    ("bcc", (3, 3, 4), 9, 2, 6, 33, 60, None),
    ("fcc", (4, 3, 4), 15, 3, 5, 64, 40, None),
    ("bcc", (4, 4, 5), 3, 5, 1, 200, 30, None),
    ("fcc", (4, 4, 4), 4, 6, 12, 150, 60, None),
    ("bcc", (4, 5, 4), 2, 10, 7, 90, 40, None),
    ("simple_cubic", (3, 4, 3), 3, 2, 9, 50, 80, None),
    ("bcc", (2, 2, 2), 3, 1, 10, 40, 150, None),
    ("fcc", (4, 4, 4), 2, 2, 6, 120, 30, 1),
    ("fcc", (5, 5, 5), 3, 2, 4, 300, 12, 2),
]


@pytest.mark.parametrize("case", CASES, ids=lambda c: f"{c[0]}-{c[1]}-s{c[2]}-sh{c[3]}-{c[5]}")
def test_rounds_match_oracle(case):
    lattice, n, ns, nsh, K, n_steps, n_iter, few = case
    V = random_V(np.random.default_rng(ns * 100 + nsh), ns, nsh, 0.06)
    setup = B.Setup(lattice, *n, ns, nsh)
    nums = equi_numbers(setup.n_atoms, ns)
    if few is not None:
        nums[-1] += nums[0] - few
        nums[0] = few
    mod = O.OracleModel(lattice, *n, V)
    runs, expect = [], []
    for seed in (31, 32):
        expect.append(mod.ns_run(O.OracleRng(seed), conc_vector(ns), nums, K, n_steps, n_iter)[:3])
        runs.append(dict(setup=setup, V=V, seed=seed, n_walkers=K, n_steps=n_steps,
                         species_concentrations=conc_vector(ns), species_numbers=nums))
    nsg = B.NestedSampling(runs)
    lim = np.concatenate([nsg.iterate(1), nsg.iterate(n_iter - 1)], axis=1)
    for k, (limits, walkers, energies) in enumerate(expect):
        assert np.array_equal(lim[k], limits)
        assert np.array_equal(nsg.energies(k), energies)
        for w in range(K):
            assert np.array_equal(nsg.walker_config(k, w), walkers[w])
