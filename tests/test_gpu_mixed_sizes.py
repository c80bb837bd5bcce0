"""Chains with fields of several sizes in one batch, more than the chip has SMs and
fewer than two for each: all of them run at once, whatever launches they come in."""
import time

import numpy as np
import pytest

import brawl_gb300 as B
from oracle import oracle as O
from tests.test_gpu_metropolis import conc_vector, random_V

pytestmark = pytest.mark.gpu

SIZES = (6, 9, 14)


def _batch(chains, V, T=4000.0):
    return B.Batch([dict(setup=B.Setup("bcc", *[SIZES[k % 3]] * 3, 4, 6), V=V, seed=500 + k,
                         beta=1.0 / (T * B.K_B_IN_RY), species_concentrations=conc_vector(4)) for k in range(chains)])


def test_mixed_sizes_match_oracle():
    V = random_V(np.random.default_rng(3), 4, 6)
    b = _batch(240, V)
    acc = b.metropolis(900)
    for k in range(0, 240, 17):
        mod = O.OracleModel("bcc", *[SIZES[k % 3]] * 3, V)
        r = O.OracleRng(500 + k)
        cfg, _ = mod.initial_setup(r, conc_vector(4))
        a, _ = mod.mc_run(cfg, r, 1.0 / (4000.0 * B.K_B_IN_RY), 900, False)
        assert acc[k] == a and np.array_equal(b.config(k), cfg), k


def test_two_chains_to_an_sm_run_at_once():
    """300 chains take little longer than 150 (1.2 times, measured); in two waves
    they took 1.8 times as long."""
    V = random_V(np.random.default_rng(3), 4, 6)

    def fastest(chains):
        b = _batch(chains, V)
        t = []
        for _ in range(9):
            t0 = time.perf_counter()
            b.metropolis(6000)
            t.append(time.perf_counter() - t0)
        b.close()
        return min(t[2:])

    assert fastest(300) < 1.5 * fastest(150)
