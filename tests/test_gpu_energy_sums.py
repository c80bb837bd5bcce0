"""total_energy's ordered sum and the initial configurations at the edges: sums
that grow through many binades, that stay near zero (energies of both signs),
that are exactly zero and of few bits (ties), lattices below, at and past the
256 terms taken at once; quotas of one atom and intervals that share a word."""
import numpy as np
import pytest

import brawl_gb300 as B
from oracle import oracle as O
from tests.test_gpu_metropolis import conc_vector, random_V

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["random", "one sign", "few bits", "zero", "tiny"])
def test_energies_at_the_edges_match_oracle(kind):
    rng = np.random.default_rng(3)
    for lattice, n, ns, nsh in [("fcc", (1, 2, 1), 2, 1), ("bcc", (4, 4, 4), 3, 2), ("fcc", (4, 4, 4), 2, 3),
                                ("bcc", (5, 5, 7), 4, 4), ("fcc", (9, 8, 11), 5, 2), ("simple_cubic", (4, 5, 6), 3, 2),
                                ("bcc", (17, 16, 15), 2, 6)]:
        V = random_V(rng, ns, nsh)
        if kind == "one sign":
            V = -np.abs(V)
        elif kind == "few bits":
            V = np.round(V * 4096.0) / 64.0
        elif kind == "zero":
            V = np.zeros_like(V)
        elif kind == "tiny":
            V = V * 1e-200
        setup = B.Setup(lattice, *n, ns, nsh)
        mod = O.OracleModel(lattice, *n, V)
        few = np.full(ns, 1, dtype=np.int64)
        few[-1] = setup.n_atoms - (ns - 1)
        chains = [dict(setup=setup, V=V, seed=60 + k, beta=1.0, species_concentrations=conc_vector(ns),
                       species_numbers=few if k == 2 else None) for k in range(3)]
        b = B.Batch(chains)
        E = b.total_energy()
        for k, c in enumerate(chains):
            cfg, _ = mod.initial_setup(O.OracleRng(60 + k), conc_vector(ns), c["species_numbers"])
            assert np.array_equal(b.config(k), cfg), (lattice, n, k)
            assert E[k] == mod.total_energy(cfg), (lattice, n, k)


@pytest.mark.parametrize("lattice,n,ns,wc", [("fcc", (1, 1, 1), 2, 1), ("bcc", (2, 1, 3), 7, 4), ("fcc", (5, 4, 6), 8, 6),
                                             ("bcc", (6, 6, 7), 15, 12), ("simple_cubic", (4, 6, 5), 9, 3)])
def test_pair_counts_at_the_edges_match_oracle(lattice, n, ns, wc):
    """Species counted in either word of eight, lattices that an offset spans,
    and shells beyond the offsets' reach."""
    V = random_V(np.random.default_rng(5), ns, 1)
    mod = O.OracleModel(lattice, *n, V)
    ch = B.Chain(B.Setup(lattice, *n, ns, 1), V)
    ch.seed(77)
    ch.initial_setup(conc_vector(ns))
    shells = ch.lattice_shells(wc)
    rho, _ = mod.radial_densities(ch.config(), shells)
    assert np.array_equal(np.asarray(ch.radial_densities(shells)), rho, equal_nan=True)


@pytest.mark.parametrize("chains", [7, 8])
def test_energies_of_few_and_many_chains_match_oracle(chains):
    """Sums of 128 to 512 terms, which few chains take 256 at a time and many one
    by one, and one term more."""
    rng = np.random.default_rng(6)
    for lattice, n, ns, nsh in [("bcc", (4, 4, 4), 3, 2), ("bcc", (5, 5, 5), 3, 4), ("fcc", (8, 4, 4), 4, 3),
                                ("bcc", (19, 3, 9), 2, 2)]:
        V = random_V(rng, ns, nsh)
        mod = O.OracleModel(lattice, *n, V)
        b = B.Batch([dict(setup=B.Setup(lattice, *n, ns, nsh), V=V, seed=60 + k, beta=1.0,
                          species_concentrations=conc_vector(ns)) for k in range(chains)])
        E = b.total_energy()
        for k in range(chains):
            assert E[k] == mod.total_energy(b.config(k)), (lattice, n, k)


@pytest.mark.parametrize("ratio", [2.0 ** 7, 2.0 ** 10, 2.0 ** 40, 1.0e200])
def test_energies_of_terms_of_two_sizes_match_oracle(ratio):
    """Some sites' energies so much larger than the others' that a sum of whole
    ulps passes 2^63 behind the first of them."""
    V = random_V(np.random.default_rng(8), 3, 2)
    V[2, 2, :] *= ratio
    mod = O.OracleModel("bcc", 8, 8, 8, V)
    few = np.array([500, 520, 4], dtype=np.int64)
    b = B.Batch([dict(setup=B.Setup("bcc", 8, 8, 8, 3, 2), V=V, seed=70 + k, beta=1.0,
                      species_concentrations=conc_vector(3), species_numbers=few if k % 2 else None) for k in range(4)])
    E = b.total_energy()
    for k in range(4):
        assert E[k] == mod.total_energy(b.config(k)), k
