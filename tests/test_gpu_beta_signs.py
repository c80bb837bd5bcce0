"""Inverse temperatures that are zero, negative, infinite or not a number, on every
kernel that a Metropolis chain may take: u < exp(-beta dE) accepts every uphill
move below zero and none that is not a number.  Against the oracle, bit for bit:
configurations, accepted moves and streams."""
import numpy as np
import pytest

import brawl_gb300 as B
from oracle import oracle as O
from tests.test_gpu_metropolis import conc_vector, random_V
from tests.test_gpu_shared_fields import _same_stream

pytestmark = pytest.mark.gpu

# lattice, n, ns, nsh, nbr_swap, depth (1: fields where they fit, 2 to 4: gathered), chains
KERNELS = [
    ("bcc", (5, 4, 6), 4, 6, False, 1, 1),
    ("bcc", (2, 3, 2), 3, 2, True, 1, 1),
    ("fcc", (5, 4, 6), 3, 3, True, 2, 1),
    ("bcc", (6, 6, 6), 4, 6, False, 3, 1),
    ("fcc", (5, 4, 6), 2, 2, False, 4, 1),
    ("bcc", (3, 4, 3), 3, 2, False, 1, 330),
    ("simple_cubic", (5, 4, 6), 3, 2, False, 1, 1),
    ("simple_cubic", (5, 4, 6), 3, 2, True, 1, 160),
    ("fcc", (38, 38, 38), 3, 2, False, 1, 1),
]


@pytest.mark.parametrize("beta", [-500.0, -1.0e-300, -0.0, 0.0, float("inf"), float("-inf"), float("nan")])
def test_any_beta_matches_oracle(beta):
    for k, (lattice, n, ns, nsh, nbr, depth, chains) in enumerate(KERNELS):
        V = random_V(np.random.default_rng(50 + k), ns, nsh)
        mod = O.OracleModel(lattice, *n, V)
        b = B.Batch([dict(setup=B.Setup(lattice, *n, ns, nsh), V=V, seed=800 + c, beta=beta, nbr_swap=nbr,
                          species_concentrations=conc_vector(ns)) for c in range(chains)])
        b.set_speculation(depth)
        acc = b.metropolis(300)
        for c in {0, chains - 1}:
            r = O.OracleRng(800 + c)
            cfg, _ = mod.initial_setup(r, conc_vector(ns))
            a, _ = mod.mc_run(cfg, r, beta, 300, nbr)
            assert acc[c] == a, (KERNELS[k], c)
            assert np.array_equal(b.config(c), cfg), (KERNELS[k], c)
            assert _same_stream(b.rng_state(c), r), (KERNELS[k], c)
