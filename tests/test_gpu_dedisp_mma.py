"""Dedispersion sums at the sizes where the tensor-core kernel's tiling can go
wrong: tile edges (2048 samples, 1 to 16 DMs per CTA, 32 channels per base fetch),
ragged DM ranges that start inside a DM block, delay spreads from none to many
steps per DM, rows that end off a 16-byte boundary, and both stages of the
subband path.  Sums are integers, so every comparison is exact."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")


def observation(nchans, nsamples, f_low=1200.0, f_high=1500.0, seed=0, levels=256):
    rng = np.random.default_rng(seed)
    freq = np.linspace(f_low, f_high, nchans) if nchans > 1 else np.array([f_low])
    return freq, rng.integers(0, levels, size=(nsamples, nchans), dtype=np.uint8)


def run(prog, data, b0, cnt):
    staged = prog.stage(torch.from_numpy(data).cuda())
    got = prog.run(staged, b0, cnt)[:, : prog.nout]
    prog.check()
    return got.cpu().numpy().view(np.uint32)


BYTES, SLICES, DENSE = 0, 1, 2

# (channels, samples, DMs, dm_low, dm_step, first DM, DM count) and the kernel
# that runs: its form and DMs per CTA
SHAPES = [
    ((61, 160001, 64, 0.0, 2.0, 8, 50), (DENSE, 8)),
    ((61, 160001, 19, 0.0, 2.0, 8, 11), (DENSE, 8)),
    ((33, 50 * 2048 + 240, 72, 0.0, 0.1, 8, 61), (DENSE, 8)),
    ((257, 75 * 2048 + 301, 56, 5.0, 0.39, 8, 48), (DENSE, 8)),
    ((40, 151 * 2048, 24, 30.0, 0.01, 8, 16), (DENSE, 8)),
    ((5, 4900037, 1, 0.5, 1.6, 0, 1), (DENSE, 8)),
    ((9, 1230003, 3, 10.0, 0.5, 0, 3), (DENSE, 8)),
    # a range that starts inside a block of 16 DMs, ragged ends
    ((8, 1420000, 25, 100.0, 80.0, 8, 17), (SLICES, 16)),
    ((8, 1420003, 25, 100.0, 30.0, 0, 25), (SLICES, 16)),
    ((12, 700000, 48, 0.0, 60.0, 8, 37), (SLICES, 16)),
    ((8, 1420000, 25, 100.0, 150.0, 8, 17), (SLICES, 8)),
    ((13, 2430011, 4, 10.0, 30.0, 0, 4), (SLICES, 4)),
    ((8, 2420000, 25, 10.0, 800.0, 8, 17), (SLICES, 4)),
    ((13, 2430011, 2, 10.0, 30.0, 0, 2), (SLICES, 2)),
    ((9, 2230003, 4, 10.0, 3000.0, 0, 4), (SLICES, 2)),
    ((9, 4230003, 2, 10.0, 12000.0, 0, 2), (SLICES, 1)),
    # too few CTAs for the tensor cores, of the program or of the range
    ((61, 60001, 19, 0.0, 2.0, 8, 11), (BYTES, 8)),
    ((64, 75 * 2048 + 77, 65, 0.0, 7.0, 16, 49), (BYTES, 8)),
    ((96, 320000, 9, 0.0, 40.0, 8, 1), (BYTES, 8)),
    ((8, 1420000, 25, 100.0, 80.0, 8, 8), (BYTES, 8)),
    ((1, 17, 1, 0.0, 1.0, 0, 1), (BYTES, 8)),
    ((300, 6161, 16, 30.0, 0.01, 0, 16), (BYTES, 8)),
]


@pytest.mark.parametrize("shape,kernel", SHAPES)
def test_sums_match_oracle(port, shape, kernel):
    from gaffa_b200 import core
    nchans, nsamples, ndm, dm_low, dm_step, b0, cnt = shape
    freq, data = observation(nchans, nsamples, seed=nchans)
    fref = float(freq.max()) if nchans > 1 else 1500.0
    tsamp = 1e-3 if nchans == 1 else 256e-6
    prog = core.DedispersionProgram(freq, nsamples, tsamp, dm_low, dm_step, ndm, ref_frequency_mhz=fref)
    assert prog.kernels(b0, cnt) == [kernel]
    want = port.dedisperse_multi_dm(data, freq, dm_low, dm_step, ndm, fref, tsamp)
    assert np.array_equal(run(prog, data, b0, cnt), want[b0:b0 + cnt])


def test_ranges_of_one_program_take_the_kernel_that_is_faster_for_them():
    """Short ranges (a candidate's 8 DMs) run on the byte kernel, long ones on
    the tensor cores, from one program's tables, with the same sums."""
    from gaffa_b200 import core
    freq, data = observation(64, 150000, seed=3)
    prog = core.DedispersionProgram(freq, 150000, 256e-6, 0.0, 1.0, 96)
    assert prog.kernels() == [(DENSE, 8)] and prog.kernels(40, 8) == [(BYTES, 8)]
    staged = prog.stage(torch.from_numpy(data).cuda())
    whole = prog.run(staged)[:, : prog.nout]
    for b0 in range(0, 96, 8):
        assert torch.equal(prog.run(staged, b0, 8)[:, : prog.nout], whole[b0:b0 + 8])
    prog.check()


@pytest.mark.parametrize("nout_mod", [-1, 0, 1, 2047])
def test_outputs_stay_inside_their_rows(nout_mod):
    """Odd row ends and an unaligned output: no sample past nout is written."""
    from gaffa_b200 import core
    freq, data = observation(40, 6000)
    probe = core.DedispersionProgram(freq, 6000, 256e-6, 0.0, 1.0, 16)
    n = 6000 - probe.nout + 150 * 2048 + nout_mod
    freq, data = observation(40, n)
    prog = core.DedispersionProgram(freq, n, 256e-6, 0.0, 1.0, 16)
    assert prog.nout == 150 * 2048 + nout_mod and prog.kernels() == [(DENSE, 8)]
    staged = prog.stage(torch.from_numpy(data).cuda())
    want = prog.run(staged)[:, : prog.nout].clone()
    stride = prog.nout + 3
    flat = torch.full((16 * stride + 1,), -7, dtype=torch.int32, device="cuda")
    out = prog.run(staged, out=flat[1:], out_stride=stride)
    prog.check()
    assert torch.equal(out[:, : prog.nout], want)
    assert bool((out[:, prog.nout:] == -7).all()) and int(flat[0]) == -7


@pytest.mark.parametrize("nbits,sbc,npn,ndm,nsamples,dm_step,kernels", [
    (2, 16, 7, 25, 30011, 0.5, [BYTES, BYTES]), (2, 64, 55, 60, 30011, 0.5, [BYTES, DENSE]),
    (8, 16, 32, 40, 30011, 0.5, [BYTES]), (2, 85, 3, 11, 30011, 0.5, [BYTES, BYTES]),
    (2, 16, 2, 40, 150011, 0.05, [DENSE, DENSE]), (2, 25, 16, 96, 200011, 8.0, [SLICES, SLICES]),
    (2, 85, 3, 41, 300011, 1.0, [SLICES, DENSE]), (2, 16, 2, 40, 150011, 6.0, [SLICES, SLICES]),
    (8, 20, 4, 64, 150011, 0.02, [DENSE]), (8, 16, 4, 64, 100003, 12.0, [SLICES])])
def test_subband_sums_match_oracle(port, nbits, sbc, npn, ndm, nsamples, dm_step, kernels):
    from gaffa_b200 import core, synth
    levels = 4 if nbits == 2 else 256
    freq, data = observation(200, nsamples, 300.0, 400.0, seed=npn, levels=levels)
    raw = synth.pack_2bit(data) if nbits == 2 else data
    prog = core.DedispersionProgram(freq, nsamples, 1e-3, 0.0, dm_step, ndm, nbits=nbits, algorithm="subband",
                                    subband_channels=sbc, ndm_per_nominal=npn)
    assert [form for form, _ in prog.kernels()] == kernels
    want = port.dedisperse_subband(data, freq, 0.0, dm_step, ndm, float(freq.max()), 1e-3, sbc, npn)
    assert np.array_equal(run(prog, raw, 0, ndm), want)
    if ndm > npn:
        assert np.array_equal(run(prog, raw, npn, ndm - npn), want[npn:])


@pytest.mark.parametrize("nbits,nsamples", [(2, 150011), (2, 150016), (8, 150001)])
def test_rows_read_as_zero_past_their_end(port, nbits, nsamples):
    """Stage one of the subband path sums windows that reach past the last
    sample, which must count as zeros whatever the staged row's padding holds."""
    from gaffa_b200 import core, synth
    freq, data = observation(96, nsamples, 300.0, 400.0, seed=7, levels=4 if nbits == 2 else 256)
    raw = synth.pack_2bit(data) if nbits == 2 else data
    prog = core.DedispersionProgram(freq, nsamples, 1e-3, 0.0, 2.0, 48, nbits=nbits, algorithm="subband",
                                    subband_channels=16, ndm_per_nominal=4)
    staged = torch.full((int(prog.info.staged_bytes),), 255, dtype=torch.uint8, device="cuda")
    got = prog.run(prog.stage(torch.from_numpy(raw).cuda(), out=staged))[:, : prog.nout]
    prog.check()
    want = port.dedisperse_subband(data, freq, 0.0, 2.0, 48, float(freq.max()), 1e-3, 16, 4)
    assert np.array_equal(got.cpu().numpy().view(np.uint32), want)


# items of (channels, samples, DMs, DM step, first DM, DM count), and how many
# take the byte kernel, slices and the dense form
@pytest.mark.parametrize("shapes,forms", [
    (((61, 160001, 24, 1.5, 8, 13), (40, 5000, 17, 1.5, 0, 17), (37, 2048 * 80, 33, 1.5, 0, 33)), [0, 0, 3]),
    (((61, 160001, 64, 2.0, 8, 50), (40, 5000, 17, 1.5, 0, 17), (8, 1420000, 25, 80.0, 8, 17)), [0, 1, 2]),
    (((8, 1420000, 25, 80.0, 8, 17), (40, 5000, 17, 1.5, 0, 17), (8, 1420003, 25, 150.0, 0, 25)), None),
    (((40, 5000, 17, 1.5, 0, 17), (25, 9000, 9, 20.0, 8, 1)), [2, 0, 0])])
def test_batch_matches_single_launches(shapes, forms):
    from gaffa_b200 import core
    items, want = [], []
    for nchans, nsamples, ndm, dm_step, b0, cnt in shapes:
        freq, data = observation(nchans, nsamples, seed=ndm)
        prog = core.DedispersionProgram(freq, nsamples, 256e-6, 0.0, dm_step, ndm)
        staged = prog.stage(torch.from_numpy(data).cuda())
        stride = (prog.nout + 3) // 4 * 4
        want.append(prog.run(staged, b0, cnt)[:, : prog.nout].clone())
        items.append((prog, staged, b0, cnt, torch.full((cnt * stride,), -1, dtype=torch.int32, device="cuda"), stride))
    batch = core.DedispersionBatch(items)
    assert sum(batch.items_per_kernel) == len(items)
    assert forms is None or batch.items_per_kernel == forms
    batch.run()
    for (prog, _, _, cnt, out, stride), w in zip(items, want):
        prog.check()
        assert torch.equal(out.view(cnt, stride)[:, : prog.nout], w)


@pytest.mark.parametrize("nbits,nchans,nsamples,begin,end", [
    (8, 132, 1000, 0, 132), (8, 132, 129, 4, 128), (8, 132, 127, 3, 130), (8, 61, 300, 0, 61),
    (2, 272, 515, 0, 272), (2, 272, 128, 16, 256), (2, 272, 131, 4, 271), (2, 20, 64, 0, 20)])
def test_staging_is_the_transpose(nbits, nchans, nsamples, begin, end):
    from gaffa_b200 import core, synth
    freq, data = observation(nchans, nsamples, seed=nsamples, levels=4 if nbits == 2 else 256)
    raw = synth.pack_2bit(data) if nbits == 2 else data
    prog = core.DedispersionProgram(freq, nsamples, 1e-3, 0.0, 0.01, 1, chan_begin=begin, chan_end=end, nbits=nbits,
                                    ref_frequency_mhz=1500.0)
    want = torch.from_numpy(np.ascontiguousarray(data[:, begin:end].T)).cuda()
    stride = int(prog.info.staged_row_stride)
    for src in (torch.from_numpy(raw).cuda(), raw):   # device input, and host input through the bounce buffer
        got = prog.stage(src).view(end - begin, stride)[:, :nsamples]
        assert torch.equal(got, want)
