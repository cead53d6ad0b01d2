"""FFA searches at the sizes where the row schedules can go wrong, against the
oracle: rows of fewer bins than wrapped samples, one lane pass with several
levels, task sizes about the one-level limit (32 rows) and about the tiles of a
CTA, odd and even level counts, one to four column passes, and large tasks that
run on the small CTAs because they are few.  Every row evaluated is a peak (the
threshold is far below), so whole transforms and S/N are compared, bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def search_both(port, shapes, widths, seed):
    """shapes: (bins, rows, rows evaluated) of the tasks of one plan."""
    from gaffa_b200 import _lib, core
    n = max(b * r for b, r, _ in shapes)
    tasks = np.zeros(len(shapes), _lib.TASK_DTYPE)
    for t, (bins, rows, rows_eval) in zip(tasks, shapes):
        t["downsample_factor"], t["effective_tsamp"] = 1.0, 1e-3
        t["input_nsamples"] = t["prepared_nsamples"] = n
        t["bins"], t["rows"], t["rows_eval"] = bins, rows, rows_eval
        t["period_begin"], t["period_end"] = bins * 1e-3, (bins + 1) * 1e-3
    x = np.random.default_rng(seed).normal(size=n).astype(np.float32)
    prog = core.FfaProgram(core.FfaPlan(tasks, widths), max_series=1)
    rec = prog.search(prog.prepare(torch.from_numpy(x).cuda().view(1, -1), 1), 1, -1e6)
    got = core.sort_peaks(prog.expand(rec))
    want = port.ffa_search(x, tasks, np.asarray(widths), snr_threshold=-1e6)
    assert len(want) == sum(e for _, _, e in shapes) * len(widths)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("bins", [2, 3, 4, 31, 32, 33, 64, 65])
def test_rows_about_every_limit(port, bins):
    rows = [1, 2, 3, 4, 5, 7, 8, 9, 15, 16, 17, 30, 31, 32, 33, 47, 63, 64, 65, 100, 127, 129]
    search_both(port, [(bins, r, r) for r in rows], [1] if bins < 5 else [1, 2, bins // 3], bins)


# tiles hold 45 to 1300 rows at these bins; 8 times more for each column pass
@pytest.mark.parametrize("bins,rows,rows_eval", [
    (2, 60000, 60000), (3, 9001, 9001), (31, 400, 400), (31, 1600, 1600), (33, 20011, 700), (120, 1500, 1500),
    (256, 800, 800), (256, 1700, 333), (256, 20003, 100), (256, 65535, 64), (512, 50, 50), (512, 3500, 400),
    (512, 40009, 50)])
def test_column_passes(port, bins, rows, rows_eval):
    search_both(port, [(bins, rows, rows_eval)], [1] if bins < 5 else [1, bins // 5], rows)


@pytest.mark.parametrize("bins,fits,large", [(64, 150, 500), (240, 45, 300), (33, 250, 2500)])
def test_few_large_tasks_among_many(port, bins, fits, large):
    search_both(port, [(bins, fits + i, fits + i) for i in range(80)] + [(bins, large, large)], [1, 3], bins)
