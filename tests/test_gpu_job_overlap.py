"""Calls made while a resident job runs asynchronously on a stream of the caller's
(a torch side stream, which does not synchronise with the default stream): the
job's results and the calls' own must be those of each alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_tracelog_lu_beside_running_job(ms, precision):
    torch = pytest.importorskip("torch")
    med = ms.Medium(3, 1200, seed=3)
    ks = 0.7 + 0.08 * np.arange(24) - 0.05j
    want, wst = ms.tracelog_batch([med], ks, precision=precision)
    mats = [ms.build_ms_matrix(ms.Medium(3, n, seed=n), 1.1 - 0.1j) for n in (40, 300)]
    alone = [ms.tracelog_lu(m) for m in mats]
    job = ms.Job("tracelog", [med], ks, precision=precision)
    side = torch.cuda.Stream()
    for _ in range(3):
        job.run(side.cuda_stream)
        beside = [ms.tracelog_lu(m) for _ in range(4) for m in mats]
        got, st = job.results()
        assert beside == 4 * alone
        assert np.array_equal(got, want) and np.array_equal(st, wst)
    job.close()


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_destroy_waits_for_a_callers_graph(ms, precision):
    """A run captured in a CUDA graph of the caller's and replayed after the job's
    results were fetched: destroying the job must wait for the replay, whose arrays
    the next job of that size is given."""
    torch = pytest.importorskip("torch")
    med = ms.Medium(3, 700, seed=4)
    ks = 0.7 + 0.02 * np.arange(100) - 0.05j
    want, _ = ms.tracelog_batch([med], ks + 0.3, precision=precision)
    for _ in range(3):
        job = ms.Job("tracelog", [med], ks, precision=precision)
        job.run()
        first, _ = job.results()
        graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
        with torch.cuda.graph(graph, stream=side):
            job.run(torch.cuda.current_stream().cuda_stream)
        graph.replay()
        again, _ = job.results()
        assert np.array_equal(first, again)
        graph.replay()
        job.close()
        nxt = ms.Job("tracelog", [med], ks + 0.3, precision=precision)
        nxt.run()
        got, st = nxt.results()
        nxt.close()
        assert np.all(st == 0) and np.array_equal(got, want)


def test_destroy_beside_a_capture(ms):
    """Destroying an idle job asks nothing of the device: a capture of the caller's
    that is under way (a job collected as garbage meanwhile) stays valid."""
    torch = pytest.importorskip("torch")
    job = ms.Job("tracelog", [ms.Medium(3, 60, seed=4)], [1.1 + 0j, 2.0 + 0j])
    job.run()
    job.results()
    x = torch.zeros(16, device="cuda")
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=side, capture_error_mode="relaxed"):
        x += 1
        job.close()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.all(x == 1)


def test_destroy_while_running(ms):
    """A job destroyed with its run in flight, the next of its size at once."""
    torch = pytest.importorskip("torch")
    med = ms.Medium(3, 700, seed=4)
    ks = 0.7 + 0.02 * np.arange(100) - 0.05j
    want, _ = ms.tracelog_batch([med], ks + 0.3)
    side = torch.cuda.Stream()
    for _ in range(3):
        job = ms.Job("tracelog", [med], ks)
        job.run(side.cuda_stream)
        job.close()
        got, st = ms.tracelog_batch([med], ks + 0.3)
        assert np.all(st == 0) and np.array_equal(got, want)
