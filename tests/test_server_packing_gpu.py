"""Windows that share a launch of the server also share the search kernel their sizes call for."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a,b,preempt_us", [
    ((571, 210, 1_000_001), (601, 210, 1_000_001), 0),                # one layout, two tensor-core sizes
    ((503, 2190, (1 << 30) - 999), (503, 2190, (1 << 30) + 1), 0),   # the second above the m of that kernel
    ((571, 210, 1_000_001), (601, 210, 1_000_001), 20_000),
])
def test_requests_of_another_kernel_take_another_launch(pg, a, b, preempt_us):
    sl, limit, inc = 4_000, 2_000_000, 300
    alone, info = [], []
    for P, d, m in (a, b):
        with pg.Job(P, d, sl, limit, max_m_inc=inc, max_m=(1 << (m + inc).bit_length()) - 1) as job:
            alone.append(job.search(m, inc))
            info.append(job.info)
    assert info[0]["limbs"] == info[1]["limbs"]
    with pg.Server(0, batch_m=8_192, max_sl=sl, slots=2 if preempt_us else 1, preempt_us=preempt_us) as srv:
        for P, d, m in ((907, 210, 1_000_001), a, b):  # tables and jobs in place
            srv.wait(srv.submit(P, d, sl, limit, m, 2))
        before = srv.stats()["launches"]
        srv.submit(907, 210, sl, limit, 1_000_001, 30_000)  # holds the slot until both requests wait
        ids = [srv.submit(P, d, sl, limit, m, inc) for P, d, m in (a, b)]
        got = [srv.wait(i) for i in ids]
        while srv.stats()["requests_done"] < 6:
            srv.next_done(1.0)
        launches = srv.stats()["launches"] - before
    for x, y in zip(alone, got):
        assert np.array_equal(x.ms, y.ms)
        assert np.array_equal(x.prev_gap, y.prev_gap) and np.array_equal(x.next_gap, y.next_gap)
    assert launches == 3
