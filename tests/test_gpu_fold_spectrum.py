"""The spectrum fold's wide and narrow forms and the projections against FP64
sums in numpy: bins at and past the wide form's limit, ragged channel counts,
several bins per sample, subints shorter than the warps' runs."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


# (samples, channels, bins, subint samples, period, start, output channels, type)
FOLDS = [(5000, 132, 96, 700, 0.2, 0, 0, np.uint8), (5000, 132, 97, 700, 0.2, 11, 0, np.uint8),
         (999, 61, 16, 1000, 0.005, 3, 0, np.uint8), (4097, 64, 32, 513, 0.31, 0, 16, np.uint8),
         (3000, 36, 64, 300, 0.017, 5, 0, np.float32), (70, 4, 8, 9, 0.05, 0, 0, np.uint8)]


@pytest.mark.parametrize("ns,nc,nbin,sub,period,start,nout,dtype", FOLDS)
def test_fold_spectrum_and_projections(ns, nc, nbin, sub, period, start, nout, dtype):
    from gaffa_b200 import _lib, core
    rng = np.random.default_rng(ns)
    x = rng.integers(0, 256, size=(ns, nc)).astype(dtype)
    cube, expo = core.fold_spectrum(torch.from_numpy(x).cuda(), period, 1e-3, nbin, sub, start, nout)
    k = nout or nc
    v = x.astype(np.float64).reshape(ns, k, nc // k).mean(2)
    nsub = -(-ns // sub)
    sums, want_e = np.zeros((nsub, nbin, k)), np.zeros((nsub, nbin))
    step = 1e-3 / period * nbin
    for t in range(ns):
        lo = (start + t) * step
        hi = lo + step
        for b in range(int(np.floor(lo)), int(np.ceil(hi))):
            w = min(hi, b + 1.0) - max(lo, float(b))
            if w > 0.0:
                sums[t // sub, b % nbin] += v[t] * w
                want_e[t // sub, b % nbin] += w
    e = want_e[:, None, :]
    want = np.where(e > 0, sums.transpose(0, 2, 1) / np.where(e > 0, e, 1.0), 0.0)
    np.testing.assert_allclose(expo.cpu().numpy(), want_e, rtol=1e-11)
    np.testing.assert_allclose(cube.cpu().numpy(), want, rtol=1e-6)   # float32 of FP64 sums: 6e-8
    prof, freq, time = (torch.empty(s, dtype=torch.float32, device="cuda") for s in ((nbin,), (k, nbin), (nsub, nbin)))
    _lib.check(_lib.lib().gf_project_folded_cube(_lib.ptr(cube), _lib.ptr(expo), nsub, k, nbin, _lib.ptr(prof),
                                                 _lib.ptr(freq), _lib.ptr(time), None))
    torch.cuda.synchronize()
    c, ex = cube.cpu().numpy().astype(np.float64), want_e.sum(0)
    ok = ex > 0
    np.testing.assert_allclose(prof.cpu().numpy()[ok], ((c * e).sum((0, 1)) / (k * np.where(ok, ex, 1)))[ok], rtol=1e-6)
    np.testing.assert_allclose(freq.cpu().numpy(), np.where(ok, (c * e).sum(0) / np.where(ok, ex, 1), 0.0), rtol=1e-6)
    np.testing.assert_allclose(time.cpu().numpy(), np.where(want_e > 0, c.mean(1), 0.0), rtol=1e-6)
