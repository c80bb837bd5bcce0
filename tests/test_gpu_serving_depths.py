"""Served anneals of lattices without fields at very high and at low temperatures,
whose rounds of trials differ, beside chains with fields and without shared memory's
kernels: each equals the oracle's run."""
import numpy as np
import pytest

from brawl_gb300 import serving as S
from tests.test_gpu_serving import _collect, _job, _oracle

pytestmark = pytest.mark.gpu


def test_served_anneals_of_any_temperature_match_oracle():
    jobs = [_job("anneal", "bcc", 22, 5, 4, 41, T_start=60000.0, delta_T=-59000.0, T_steps=2, sweeps_per_T=1),
            _job("anneal", "bcc", 23, 4, 6, 42, T_start=800.0, delta_T=-100.0, T_steps=2, sweeps_per_T=1),
            _job("anneal", "fcc", 17, 4, 2, 43, T_start=4000.0, delta_T=-1500.0, T_steps=2, sweeps_per_T=1),
            _job("anneal", "bcc", 4, 2, 2, 44, T_start=30000.0, delta_T=-100.0, T_steps=2, sweeps_per_T=30),
            _job("anneal", "fcc", 3, 5, 6, 45, T_start=900.0, delta_T=-100.0, T_steps=2, sweeps_per_T=30)]
    with S.Server(max_trials=9000) as srv:
        ids = [srv.submit(j) for j in jobs]
        got = [_collect(srv, k) for k in ids]
    for job, r in zip(jobs, got):
        values, cfg = _oracle(job)
        assert np.array_equal(r["values"], values), job["L"]
        assert np.array_equal(r["config"], cfg), job["L"]
