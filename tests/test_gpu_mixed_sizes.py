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


@pytest.mark.parametrize("chains", [150, 200])
def test_very_hot_chains_beside_cool_ones_match_oracle(chains):
    """One and two chains to an SM, every second one at an infinite temperature
    (which gather their sums where two share an SM), in calls at two temperatures
    and with classes of their own."""
    V = random_V(np.random.default_rng(4), 3, 2)
    T = np.where(np.arange(chains) % 2, 400.0, 1.0e7)
    mod = O.OracleModel("bcc", 5, 5, 5, V)
    b = B.Batch([dict(setup=B.Setup("bcc", 5, 5, 5, 3, 2), V=V, seed=90 + k, beta=1.0 / (T[k] * B.K_B_IN_RY),
                      nbr_swap=k % 3 == 0, species_concentrations=conc_vector(3)) for k in range(chains)])
    acc = b.metropolis(400)
    b.set_beta(1.0 / (T[::-1] * B.K_B_IN_RY))
    acc = acc + b.metropolis(401)
    b.set_class_depths([1])
    acc = acc + b.metropolis(402)
    for k in (0, 1, 2, 3, chains - 2, chains - 1):
        r = O.OracleRng(90 + k)
        cfg, _ = mod.initial_setup(r, conc_vector(3))
        a = sum(mod.mc_run(cfg, r, 1.0 / (t * B.K_B_IN_RY), n, k % 3 == 0)[0]
                for t, n in ((T[k], 400), (T[::-1][k], 401), (T[::-1][k], 402)))
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


def test_a_few_long_chains_among_many_short_ones_match_oracle():
    """Trials in proportion to the sites: the short chains wait for a place."""
    V = random_V(np.random.default_rng(5), 4, 6)
    b = _batch(240, V, 1500.0)
    trials = np.array([s.n_atoms // 4 for s in b.setups])
    acc = b.metropolis(trials)
    for k in range(0, 240, 23):
        mod = O.OracleModel("bcc", *[SIZES[k % 3]] * 3, V)
        r = O.OracleRng(500 + k)
        cfg, _ = mod.initial_setup(r, conc_vector(4))
        a, _ = mod.mc_run(cfg, r, 1.0 / (1500.0 * B.K_B_IN_RY), int(trials[k]), False)
        assert acc[k] == a and np.array_equal(b.config(k), cfg), k
