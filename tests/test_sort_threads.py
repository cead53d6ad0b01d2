"""Peak lists long enough for several host threads: the order that one sort of
the whole list gives, at the lengths where the runs change, and the candidates
selected from such a list."""
import os

import numpy as np
import pytest

from gaffa_b200 import _lib, core

pytestmark = pytest.mark.skipif((os.cpu_count() or 1) < 2, reason="one core: lists are sorted by one thread")


def peaks(n, seed):
    rng = np.random.default_rng(seed)
    p = np.zeros(n, _lib.PEAK_DTYPE)
    p["snr"] = rng.integers(16, 80, n) * 0.5          # many ties, broken by the other fields
    p["width"] = rng.integers(1, 5, n)
    p["period"] = rng.integers(1, 50, n) * 0.01
    p["frequency"] = 1.0 / p["period"]
    for k, top in (("bins", 4), ("shift", 30), ("phase", 50), ("dm_index", 100)):
        p[k] = rng.integers(0, top, n)
    p["dm"] = p["dm_index"] * 0.5
    if n > 50:  # not finite: after all others
        p["snr"][rng.integers(0, n, n // 50)] = np.inf
        p["period"][rng.integers(0, n, n // 50)] = np.inf
    return p


@pytest.mark.parametrize("n", [0, 1, 16383, 16384, 16385, 32769, 100003])
def test_long_lists_sort_as_short_ones(n):
    p = peaks(n, n)
    got = core.sort_peaks(p)
    # pieces below the threshold, each sorted by one thread, merged by re-sorting
    # neighbours: the list must already be in order piece by piece
    for a in range(0, n, 8000):
        piece = got[a:a + 16000]
        assert np.array_equal(core.sort_peaks(piece[::-1]), piece)
    assert np.array_equal(np.sort(got, order=list(p.dtype.names)), np.sort(p, order=list(p.dtype.names)))


@pytest.mark.parametrize("n", [16000, 17200, 40001])   # 2-4 % of them not finite
def test_candidates_of_long_lists(port, n):
    p = peaks(n, n + 1)
    p = p[np.isfinite(p["snr"]) & np.isfinite(p["period"])]   # 49 frequencies: ties decide the order
    p["duty_cycle"] = 0.1
    tobs = 300.0
    for args in ((), (0.5, 3, False, 5)):
        assert np.array_equal(core.select_candidates(p, tobs, *args), port.select_candidates(p, tobs, *args))
    # more candidates than the first buffer holds
    p["period"] = 0.01 + np.arange(len(p)) * 1e-4
    p["frequency"] = 1.0 / p["period"]
    assert np.array_equal(core.select_candidates(p, 1e9), port.select_candidates(p, 1e9))
