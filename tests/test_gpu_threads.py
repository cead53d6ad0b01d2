"""Calls from several threads whose launches want different amounts of shared
memory: a kernel's limit must not depend on the call, or one thread lowers it
under another's launch."""
import threading

import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def side_by_side(calls, repeats):
    """Each call over and over on a thread and stream of its own."""
    errors = []

    def work(call):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(repeats):
                    call()
                torch.cuda.current_stream().synchronize()
        except Exception as e:
            errors.append(e)

    torch.cuda.synchronize()
    threads = [threading.Thread(target=work, args=(c,)) for c in calls]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


def test_folds_of_different_bins():
    from gaffa_b200 import _lib
    x = torch.arange(4096, dtype=torch.int32, device="cuda")

    def fold(nbin):
        n = int(_lib.lib().gf_fold_workspace_bytes(4096, nbin))
        ws = torch.empty(n, dtype=torch.uint8, device="cuda")
        prof = torch.empty(nbin, dtype=torch.float32, device="cuda")
        expo = torch.empty(nbin, dtype=torch.float64, device="cuda")
        return lambda: _lib.check(_lib.lib().gf_fold_time_series(
            _lib.ptr(x), 1, 4096, 0.5, 1e-3, nbin, 0, _lib.ptr(prof), _lib.ptr(expo), _lib.ptr(ws),
            torch.cuda.current_stream().cuda_stream))

    side_by_side([fold(16), fold(8192), fold(64), fold(4096)], 4000)


def test_prepares_of_different_downsampling():
    from gaffa_b200 import _lib, core

    def prepare(pmin, pmax):
        n = 60000
        ffa = core.FfaProgram(core.make_riptide_ffa_plan(n, 1e-3, pmin, pmax, bins_min=4, bins_max=5), max_series=1)
        series = torch.from_numpy(np.random.default_rng(1).normal(size=(1, n)).astype(np.float32)).cuda()
        stats = torch.tensor([[0.0, 1.0]], dtype=torch.float64, device="cuda")
        out = torch.zeros(1, ffa.prepared_floats, device="cuda")
        want = ffa.prepare(series, 1, stats, out=out).clone()
        call, args = _lib.lib().gf_ffa_prepare, (ffa._h, _lib.ptr(series), 1, n, _lib.ptr(stats), _lib.ptr(out))
        return lambda: _lib.check(call(*args, torch.cuda.current_stream().cuda_stream)), out, want, (ffa, series, stats)

    cases = [prepare(0.05, 0.1), prepare(10.0, 20.0), prepare(0.05, 0.2), prepare(5.0, 25.0)]
    side_by_side([c[0] for c in cases], 4000)
    for _, out, want, _ in cases:
        assert torch.equal(out, want)
