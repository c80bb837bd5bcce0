"""Nested-sampling walks of compositions with a scarce species, whose second sites
are drawn again hundreds of times a step, across the ends of what is looked at at
once: against the oracle, bit for bit."""
import numpy as np
import pytest

import brawl_gb300 as B
from oracle import oracle as O
from tests.test_gpu_metropolis import random_V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,n,nsh,numbers,steps,iters", [
    ("fcc", (8, 8, 8), 2, (1, 2047), 40, 6),
    ("fcc", (8, 8, 8), 3, (2027, 21), 120, 12),
    ("bcc", (9, 10, 11), 4, (1960, 19, 1), 90, 10),
    ("simple_cubic", (6, 5, 7), 2, (5, 1670, 5), 90, 8),
    ("fcc", (6, 6, 6), 6, (60, 804), 200, 20),
])
def test_scarce_species_match_oracle(lattice, n, nsh, numbers, steps, iters):
    ns = len(numbers)
    V = random_V(np.random.default_rng(17), ns, nsh, 0.06)
    setup = B.Setup(lattice, *n, ns, nsh)
    nums = np.array(numbers, dtype=np.int64)
    assert nums.sum() == setup.n_atoms
    conc = np.concatenate([[0.0], nums / nums.sum()])
    mod = O.OracleModel(lattice, *n, V)
    runs, expect = [], []
    for seed in (5, 6, 7):
        expect.append(mod.ns_run(O.OracleRng(seed), conc, nums, 4, steps, iters)[:3])
        runs.append(dict(setup=setup, V=V, seed=seed, n_walkers=4, n_steps=steps, species_concentrations=conc,
                         species_numbers=nums))
    r = B.NestedSampling(runs)
    lim = np.concatenate([r.iterate(1), r.iterate(iters - 1)], axis=1)
    for k, (limits, walkers, energies) in enumerate(expect):
        assert np.array_equal(lim[k], limits)
        assert np.array_equal(r.energies(k), energies)
        for w in range(4):
            assert np.array_equal(r.walker_config(k, w), walkers[w])
