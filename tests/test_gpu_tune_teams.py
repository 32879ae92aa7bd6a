"""What a tuning entry reaches: one CTA per SM is a choice for batches that fill the
chip, so a single matrix keeps its cluster; and the FP64 engine's one launch above
96 rows is timed once and leaves the table's CTA count alone."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _seconds(f):
    f()
    best = 1e9
    for _ in range(5):
        t = time.perf_counter()
        f()
        best = min(best, time.perf_counter() - t)
    return best


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_one_matrix_keeps_its_cluster(ms, precision):
    med = ms.Medium(3, 700, seed=6)
    k = np.array([1.3 - 0.1j])
    want, _ = ms.tracelog_batch([med], k, precision=precision)
    base = _seconds(lambda: ms.tracelog_batch([med], k, precision=precision))
    ms.tune_set("tracelog", precision, 700, None, 1)
    try:
        got, st = ms.tracelog_batch([med], k, precision=precision)
        tuned = _seconds(lambda: ms.tracelog_batch([med], k, precision=precision))
    finally:
        ms.tune_set("tracelog", precision, 700, None, 0)
    assert np.all(st == 0) and np.array_equal(got, want)
    assert tuned < 1.4 * base  # (a CTA alone takes over twice as long)


def test_autotune_above_96_rows(ms):
    try:
        times, choice = ms.autotune("tracelog", "fp64", 3, 110, nitem=ms.sm_count())
        assert set(times) == {"fp64 x1"} and times["fp64 x1"] > 0 and choice == ("fp64", 0)
        times, choice = ms.autotune("tracelog", "mixed", 3, 110, nitem=2 * ms.sm_count())
        assert set(times) == {"fp64 x1", "mixed x1", "mixed x2"} and all(t > 0 for t in times.values())
        best = min(times, key=times.get)
        assert choice == (best.split()[0], 0 if best[0] == "f" else int(best[-1]))
    finally:
        ms.tune_set("tracelog", "mixed", 110, None, 0)
        ms.tune_set("tracelog", "fp64", 110, None, 0)
    assert ms.tune_table() == []
