"""A call that the device-memory budget refused is made again on the same context: it is refused again,
or gives the right values; never values from tables that the first call left unfinished.  The budgets
step through the allocations of the analytic stage one after the other."""
import numpy as np
import pytest

from slater_stoch_gb300 import api, basis, configs
from slater_stoch_gb300._lib import SSError

pytestmark = pytest.mark.gpu


def test_refused_analytic_stage_can_be_retried():
    b = configs.h2o_minimal(ng0=3)
    q = basis.build_mapping(b.n)
    with api.Context(0) as ctx:
        ctx.set_basis(b)
        ctx.set_quartets(*q)
        ref, _ = ctx.gauss_eri()
    refused = done = 0
    for budget in range(16 << 10, 3 << 20, 24 << 10):
        with api.Context(0, budget) as ctx:
            for _ in range(3):
                try:
                    ctx.set_basis(b)
                    ctx.set_quartets(*q)
                    g, _ = ctx.gauss_eri()
                except SSError as e:
                    assert "budget" in str(e)
                    refused += 1
                    continue
                np.testing.assert_array_equal(g, ref)
                done += 1
    assert refused >= 30 and done >= 3
