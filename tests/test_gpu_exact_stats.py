"""Statistics of detrended series: the parallel FP64 sums must have the bits of
the sequential loop, on series whose sums are all exact, exact up to some
segment (16384 samples), never exact, and not finite."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def sequential_stats(y):
    y = y.astype(np.float64)
    total, sq = np.cumsum(y)[-1], np.cumsum(y * y)[-1]     # cumsum adds one by one
    n = float(len(y))
    mean = total / n
    var = sq / n - mean * mean
    return mean, 1.0 / np.sqrt(var)


def series(kind, n, rng):
    if kind == "u32":                                      # dedispersed sums: exact throughout
        return (rng.normal(size=n) * 256 + 32768).round().astype(np.int32)
    if kind == "loud":                                     # sums of squares outgrow 53 bits part way
        return (rng.normal(size=n) * 20000 + 600000).round().astype(np.int32)
    return (rng.normal(size=n) * 3).astype(np.float32)     # 24 bits per sample: rounds at once


@pytest.mark.parametrize("kind", ["u32", "loud", "f32"])
@pytest.mark.parametrize("n,stride", [(16384 * 2, 16384 * 2), (16384 * 3 + 5, 16384 * 3 + 8), (40003, 40003),
                                      (5000, 5003), (16383, 16384)])
def test_stats_have_the_sequential_bits(kind, n, stride):
    from gaffa_b200 import core
    rng = np.random.default_rng(n)
    x = np.stack([np.resize(series(kind, n, rng), stride) for _ in range(3)])
    pre = core.PreprocessProgram(n, 1e-3, window_seconds=0.5, min_points=101, max_series=3)
    t = torch.from_numpy(x).cuda()
    stats = pre.run(t).cpu().numpy()
    pre.synchronize()
    y = t.view(torch.float32).cpu().numpy()[:, :n]
    for got, row in zip(stats, y):
        assert tuple(got) == sequential_stats(row)


@pytest.mark.parametrize("nseries", [1184, 1185, 1190, 1203])
def test_many_series_share_ctas(nseries):
    """Launches of more than 1184 series of floats take four to a CTA, also where
    the last CTA has fewer, with sums that are exact, exact part way and never
    exact side by side; so do batches of that many in all."""
    from gaffa_b200 import core
    n = 16384 + 700
    rng = np.random.default_rng(nseries)
    x = np.stack([series(("u32", "loud")[k % 2], n, rng) for k in range(8)])[rng.integers(0, 8, nseries)]
    f = np.stack([series("f32", n, rng) if k % 2 else series("u32", n, rng).astype(np.float32)
                  for k in range(8)])[rng.integers(0, 8, nseries)]
    parts = []
    for data in (x, f):
        pre = core.PreprocessProgram(n, 1e-3, window_seconds=0.5, min_points=101, max_series=nseries)
        t = torch.from_numpy(data).cuda()
        stats = pre.run(t).cpu().numpy()
        pre.synchronize()
        y = t.view(torch.float32).cpu().numpy()
        done = {}
        for got, row in zip(stats, y):
            key = row.tobytes()
            if key not in done:
                done[key] = sequential_stats(row)
            assert tuple(got) == done[key]
        parts.append((data, y, stats))
    # as two pieces of a batch
    cut = 600
    for data, want, want_stats in parts:
        pres = [core.PreprocessProgram(n, 1e-3, window_seconds=0.5, min_points=101, max_series=m)
                for m in (cut, nseries - cut)]
        bufs = [torch.from_numpy(np.ascontiguousarray(d)).cuda() for d in (data[:cut], data[cut:])]
        core.PreprocessBatch((p, b, b.shape[0]) for p, b in zip(pres, bufs)).run()
        for p in pres:
            p.synchronize()
        assert np.array_equal(np.concatenate([b.view(torch.float32).cpu().numpy() for b in bufs]), want)
        assert np.array_equal(np.concatenate([p.stats[: b.shape[0]].cpu().numpy() for p, b in zip(pres, bufs)]),
                              want_stats)


@pytest.mark.parametrize("u32", [False, True])
def test_medians_of_many_series(u32):
    """Short windows slide where the series fill the GPU: the same medians."""
    from gaffa_b200 import core
    rng = np.random.default_rng(4)
    n, m, w = 700, 5000, 101
    base = rng.integers(-500, 500, size=(16, n)) + (100000 if u32 else 0)
    pick = rng.integers(0, 16, m)
    x = base[pick].astype(np.int32 if u32 else np.float32)
    t = torch.from_numpy(x).cuda()
    pre = core.PreprocessProgram(n, 1.0, window_seconds=float(w), min_points=w, max_series=m)
    pre.run(t)
    padded = np.pad(base.astype(np.float32), ((0, 0), (w // 2, w // 2)), mode="edge")
    med = np.median(np.lib.stride_tricks.sliding_window_view(padded, w, axis=1), axis=2).astype(np.float32)
    assert np.array_equal(t.view(torch.float32).cpu().numpy(), x.astype(np.float32) - med[pick])


def test_nonfinite_after_an_exact_segment():
    from gaffa_b200 import core
    x = np.random.default_rng(1).normal(size=(1, 50000)).astype(np.float32)
    x[0, 40000] = np.inf
    pre = core.PreprocessProgram(50000, 1e-3, window_seconds=0.5, min_points=101, max_series=1)
    pre.run(torch.from_numpy(x).cuda())
    with pytest.raises(ValueError, match="finite"):
        pre.synchronize()


@pytest.mark.parametrize("w", [1, 3, 5, 63, 101, 127, 129, 255])
@pytest.mark.parametrize("n", [600, 513, 2049])
def test_running_median_at_every_window_form(w, n):
    """Selected (to 127 samples) and sliding medians of an edge-padded series."""
    from gaffa_b200 import core
    rng = np.random.default_rng(w * n)
    x = np.stack([rng.normal(size=n), rng.integers(-3, 4, size=n), np.linspace(-1e6, 1e6, n)]).astype(np.float32)
    pre = core.PreprocessProgram(n, 1.0, window_seconds=float(w), min_points=w, max_series=3, reject_constant=False)
    assert int(pre.info.scrunch_factor) == 1
    t = torch.from_numpy(x.copy()).cuda()
    pre.run(t)
    padded = np.pad(x, ((0, 0), (w // 2, w // 2)), mode="edge")
    med = np.median(np.lib.stride_tricks.sliding_window_view(padded, w, axis=1), axis=2).astype(np.float32)
    assert np.array_equal(t.cpu().numpy(), x - med)
