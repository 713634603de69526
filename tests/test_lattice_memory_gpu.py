"""The primes' lattices are kept only in memory that nothing else asks for."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _free() -> int:
    return torch.cuda.mem_get_info()[0]


def test_lattices_give_way_to_another_job(pg):
    """A job that fits beside another one's prime tables, but not beside its lattices too, is created."""
    a_args = dict(p=503, d=2190, sl=10_000, max_prime=2_000_000_000, max_m_inc=1_500, max_m=2_000_000)
    b_args = dict(p=337, d=2310, sl=7_500, max_prime=2_000_000_000, max_m_inc=1_500, max_m=11_000_000)
    fill = None
    with pg.Job(**b_args, flags=pg.PG_JOB_COMPACT_WALK) as job:
        b_rows = job.sieve_interval(10_000_000, 1_500)[1]
        lat = 16 * job.info["num_primes"]
    torch.cuda.empty_cache()
    with pg.Job(**a_args) as a:
        held = a.info["device_bytes"]
        assert held > 28 * a.info["num_primes"]  # 12 B a prime and its lattice
        a_ms, a_rows = a.sieve_interval(1_000_000, 1_500)
        need = 12 * (lat // 16) + 300_000_000    # B's tables and buffers
        try:
            fill = torch.empty(_free() - need + 600_000_000, dtype=torch.uint8, device="cuda")
            with pg.Job(**b_args, flags=pg.PG_JOB_COMPACT_WALK) as b:
                assert np.array_equal(b.sieve_interval(10_000_000, 1_500)[1], b_rows)
                ms, rows = a.sieve_interval(1_000_000, 1_500)
                assert np.array_equal(ms, a_ms) and np.array_equal(rows, a_rows)  # by search, without lattices
                gaps = a.search(1_000_000, 1_500)
        finally:
            del fill
            torch.cuda.empty_cache()
        assert np.array_equal(gaps.ms, a_ms) and (gaps.next_gap > 0).all()


def test_compact_walk_jobs_keep_no_lattices(pg):
    args = dict(p=337, d=2310, sl=7_500, max_prime=100_000_000, max_m_inc=10_000, max_m=11_000_000)
    with pg.Job(**args, flags=pg.PG_JOB_COMPACT_WALK) as job:
        compact, primes = job.info["device_bytes"], job.info["num_primes"]
        rows = job.sieve_interval(10_000_000, 300)[1]
    with pg.Job(**args) as job:
        assert job.info["device_bytes"] - compact >= 16 * primes
        assert np.array_equal(job.sieve_interval(10_000_000, 300)[1], rows)


def test_server_lattices_give_way_to_tables(pg):
    """A budget that holds seven table sets holds all of them, though the first set found room for its lattices."""
    keys = [(337, d) for d in (2310, 210, 30, 6)] + [(331, d) for d in (2310, 210, 30)]
    limit, knobs = 100_000_000, dict(batch_m=4_096, window_m=4_096, max_windows=4, max_sl=2_000)
    with pg.Server(0, **knobs) as srv:
        slots = srv.stats()["resident_bytes"]
    with pg.Job(337, 2310, 2_000, limit, max_m_inc=64, max_m=11_000_000) as job:
        primes = job.info["num_primes"]
    one = 12 * primes + (1 << 20)                      # a set's tables and its job
    estimate = int(15.12 * limit / 18.42) + (2 << 20)  # what the server reserves before it builds one
    with pg.Server(0, hbm_budget=slots + 6 * one + estimate + (16 << 20), **knobs) as srv:
        for P, d in keys:
            res = srv.wait(srv.submit(P, d, 2_000, limit, 10_000_001, 40))
            assert (res.next_gap > 0).all()
            if (P, d) == keys[0]:
                assert srv.stats()["resident_bytes"] - slots > 28 * primes
        st = srv.stats()
    assert st["tables_built"] == len(keys) and st["tables_evicted"] == 0


def test_lattices_give_way_beside_searches_in_flight(pg):
    """Another thread's windows keep their results while the lattices they read are freed between launches."""
    import threading
    a_args = dict(p=503, d=2190, sl=10_000, max_prime=1_000_000_000, max_m_inc=1_500, max_m=2_000_000)
    b_args = dict(p=337, d=2310, sl=7_500, max_prime=1_000_000_000, max_m_inc=1_500, max_m=11_000_000,
                  flags=pg.PG_JOB_COMPACT_WALK)
    results, stop, errors = [], threading.Event(), []

    def search(job):
        try:
            while not stop.is_set():
                tickets = [job.submit(1_000_000, 1_500) for _ in range(2)]
                results.extend(job.wait(t) for t in tickets)
        except Exception as e:  # noqa: BLE001 -- reported by the main thread
            errors.append(e)

    torch.cuda.empty_cache()
    fill = None
    with pg.Job(**a_args) as a:
        first = a.search(1_000_000, 1_500)
        worker = threading.Thread(target=search, args=(a,))
        worker.start()
        try:
            need = 12 * a.info["num_primes"] + 300_000_000
            fill = torch.empty(_free() - need + 400_000_000, dtype=torch.uint8, device="cuda")
            with pg.Job(**b_args) as b:
                assert (b.search(10_000_000, 1_500).next_gap > 0).all()
                while len(results) < 12 and not errors:
                    stop.wait(0.05)
        finally:
            stop.set()
            worker.join()
            del fill
            torch.cuda.empty_cache()
    assert not errors and len(results) >= 12
    for r in results:
        assert np.array_equal(r.prev_gap, first.prev_gap) and np.array_equal(r.next_gap, first.next_gap)
