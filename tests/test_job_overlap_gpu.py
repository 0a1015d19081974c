"""ss_two_e_job queues its MC while the analytic stage runs, also where the uploads of both wrap the
staging ring: the first MC launch is queued within half of the stage's own time, on a new basis and on
a resident one, whatever fill of the ring a job finds."""
import threading
import time

import pytest

from slater_stoch_gb300 import api, basis, configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("new_basis", [True, False])
def test_the_mc_is_queued_beside_the_analytic_stage(new_basis):
    b = configs.h2o_26(ng0=20)
    q = basis.build_mapping(b.n)
    job = lambda ctx: ctx.two_e_job(1.8, 3, 1 << 14, 2, "shared", "split_bf16")  # noqa: E731
    with api.Context(0) as ctx:
        ctx.set_basis(b)
        ctx.set_quartets(*q)
        job(ctx)
        ctx.invalidate()
        n0, t0 = ctx.launches, time.perf_counter()
        ctx.gauss_eri()
        stage, launches = time.perf_counter() - t0, ctx.launches - n0
        late = []
        for _ in range(8):
            if new_basis:
                ctx.set_basis(b)
                ctx.set_quartets(*q)
            n0, t0 = ctx.launches, time.perf_counter()
            worker = threading.Thread(target=job, args=(ctx,))
            worker.start()
            while ctx.launches - n0 <= launches and worker.is_alive():
                time.sleep(0.0002)
            late.append(time.perf_counter() - t0)
            worker.join()
        # measured 7 to 10 ms of 47; one of the eight may meet a busy host
        assert sorted(late)[-2] <= 0.5 * stage, (late, stage)
