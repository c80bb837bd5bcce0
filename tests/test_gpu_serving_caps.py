"""The server's own limits on resident walkers' jobs and runs: a nested-sampling run in
rounds holds an SM, so 48 are resident at most unless the caller says otherwise."""
import pytest

from brawl_gb300 import serving as S
from tests.test_gpu_serving import _job

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cap,at_most", [(0, 48), (50, 50)])
def test_nested_runs_beyond_the_cap_wait_for_an_end(cap, at_most):
    with S.Server(max_active_ns=cap) as srv:
        ids = [srv.submit(_job("ns", "fcc", 2, 3, 2, 31 + k, ns_walkers=16, ns_steps=400, ns_iter=800))
               for k in range(at_most + 4)]
        got = [srv.wait(i, timeout=300) for i in ids]
    assert all(r["status"] == 0 for r in got)
    first_end = min(r["t_finish"] for r in got)
    assert sum(r["t_admit"] < first_end for r in got) == at_most
