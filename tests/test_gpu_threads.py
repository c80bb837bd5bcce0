"""Batches of several sizes that run one kernel, each called from a thread of its
own: no launch meets an attribute that another thread set for a smaller one, and
each batch's chains are those of its calls alone."""
import threading

import numpy as np
import pytest

import brawl_gb300 as B
from oracle import oracle as O
from tests.test_gpu_metropolis import conc_vector, random_V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lattice,sizes,ns,nsh,depth", [
    ("bcc", (5, 15, 7, 12), 4, 6, 1),               # fields
    ("bcc", (5, 15, 7, 12), 4, 6, 3),               # gathered
    ("simple_cubic", (4, 12, 6, 10), 3, 2, 1),      # rounds of trials
])
def test_batches_on_threads_match_oracle(lattice, sizes, ns, nsh, depth):
    V = random_V(np.random.default_rng(2), ns, nsh)
    beta = 1.0 / (1200.0 * B.K_B_IN_RY)
    batches, calls, faults = [], 1500, []
    for L in sizes:
        b = B.Batch([dict(setup=B.Setup(lattice, L, L, L, ns, nsh), V=V, seed=30 + L, beta=beta,
                          species_concentrations=conc_vector(ns))])
        b.set_speculation(depth)
        batches.append(b)

    def run(b):
        try:
            for _ in range(calls):
                b.metropolis(3)
        except B.BrawlError as e:
            faults.append(str(e))

    threads = [threading.Thread(target=run, args=(b,)) for b in batches]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not faults
    for L, b in zip(sizes, batches):
        mod, r = O.OracleModel(lattice, L, L, L, V), O.OracleRng(30 + L)
        cfg, _ = mod.initial_setup(r, conc_vector(ns))
        mod.mc_run(cfg, r, beta, 3 * calls, False)
        assert np.array_equal(b.config(0), cfg), L
