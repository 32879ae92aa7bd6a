"""Failure path of the FP64 engine's tensor-core updates (items of n > 96): the
first operand wait of each update is given a limit of zero polls, so it runs out
at once.  The engine must issue no MMA, report MSGPU_S_TIMEOUT (value NaN) for
every item, free its tensor memory and return; the next run on the same context
must be correct."""
import numpy as np
import pytest

from helpers import rel

pytestmark = pytest.mark.gpu

S_TIMEOUT = 8


@pytest.mark.parametrize("nitem", [1, 20, 400])  # a cluster on one matrix, small teams, more items than SMs
def test_first_operand_wait_timeout(ms, oracle, nitem):
    n = 129
    med = ms.Medium(3, n, seed=5)
    ks = 0.6 + 2.3 * np.arange(nitem) / max(1, nitem - 1) - 0.1j
    for batch in (ms.tracelog_batch, ms.dk_log_det_batch):
        want, st = batch([med], ks)
        assert np.all(st == 0)
        ms.debug_first_wait_limit(0)
        try:
            got, st = batch([med], ks)
        finally:
            ms.debug_first_wait_limit(-1)
        assert np.all(st & S_TIMEOUT), st
        assert np.all(np.isnan(got.real))
        got, st = batch([med], ks)
        assert np.all(st == 0) and np.array_equal(got, want)
    want, _ = oracle.tracelog_batch(3, n, med.pos, ks[:1])
    got, _ = ms.tracelog_batch([med], ks)
    assert rel(got[0].real, want[0].real) < 1e-11


def test_tracelog_lu_timeout_raises(ms):
    small, big = (ms.build_ms_matrix(ms.Medium(3, n, seed=2), 1.2 - 0.1j) for n in (96, 150))
    want = [ms.tracelog_lu(small), ms.tracelog_lu(big)]
    ms.debug_first_wait_limit(0)
    try:
        with pytest.raises(ms.MsgpuError):
            ms.tracelog_lu(big)
        assert ms.tracelog_lu(small) == want[0]  # no device waits below 97 rows
    finally:
        ms.debug_first_wait_limit(-1)
    assert [ms.tracelog_lu(small), ms.tracelog_lu(big)] == want


def test_graph_run_follows_the_limit(ms):
    med = ms.Medium(3, 129, seed=5)
    ks = 0.6 + 0.1 * np.arange(8) - 0.1j
    job = ms.Job("tracelog", [med], ks)
    job.use_graph(True)
    job.run()
    want, st = job.results()
    assert np.all(st == 0)
    ms.debug_first_wait_limit(0)
    try:
        job.run()
        _, st = job.results()
        assert np.all(st & S_TIMEOUT)
    finally:
        ms.debug_first_wait_limit(-1)
    job.run()
    got, st = job.results()
    assert np.all(st == 0) and np.array_equal(got, want)
    job.close()
