"""Dedispersion sums against the oracle where the layouts and staged kernels can go wrong:
column counts around the folded segments and block tiles, rows around the row groups,
subbands around the field and packing limits at full-scale samples, channel counts off
the load words, band starts, RFI stages per folded segment, and plans whose delays are
too long for the fold (time-order kernels).  Sums are whole numbers: equality."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from astroflow_b200.dedisp import Batch, IqrmParams, Plan, RfiParams  # noqa: E402
from oracle import oracle as O  # noqa: E402

F32 = np.float32


def to_np(t):
    return t.view(torch.int32).cpu().numpy().view(np.uint32)


def dev(x):
    return torch.from_numpy(x.view(np.int16) if x.dtype == np.uint16 else x).cuda().view(
        torch.uint16 if x.dtype == np.uint16 else torch.uint8)


def data(n, nchans, nbits, full=False):
    rng = np.random.default_rng(n * 31 + nchans)
    dt = np.uint8 if nbits == 8 else np.uint16
    top = 2 ** nbits - 1
    x = rng.integers(0, top + 1, size=(n, nchans)).astype(dt)
    if full:
        x[rng.random((n, nchans)) < 0.97] = top
    return x


def subband(n, nchans, nbits, hi, step, ds, width, band, zdm, iqrm, tsamp=64e-6, full=False):
    x = data(n, nchans, nbits, full)
    foff = float(F32(300.0 / nchans))
    hdr = dict(tsamp=float(F32(tsamp)), fch1=1150.0, foff=foff, nbits=nbits, nchans=nchans, ndata=n)
    freq = O.freq_table_header(hdr["fch1"], hdr["foff"], nchans)
    f0, f1 = freq[0] + band * (freq[-1] - freq[0]), freq[-1]
    fs, fe = float(F32(f0)), float(F32(f1))
    iq = IqrmParams(mode=1, radius_frac=0.1, nsigma=3.0, win_sec=n * tsamp * 0.4, hop_sec=n * tsamp * 0.2)
    plan = Plan(hdr, 0.0, hi, fs, fe, step, ds, algorithm="subband", subband_width=width,
                zero_dm_mode="range" if zdm else "callsite",
                rfi=RfiParams(use_zero_dm=zdm, use_iqrm=iqrm, iqrm=iq, use_mask=True), bad_channels=[1, nchans // 2])
    ref = x.copy()
    if ds > 1:
        ref = O.time_binning(ref, nchans, ds)
    cs, ce = plan.info["chan_start"], plan.info["chan_end"]
    if iqrm:
        t0, t1, masks = O.iqrm_masks(ref, nchans, cs, ce, float(F32(F32(tsamp) * F32(ds))), iq)
        O.apply_window_masks(ref, nchans, t0, t1, masks)
    if zdm:
        O.zero_dm_range_exact(ref, nchans, cs, ce)
    O.mark_channels(ref, nchans, [1, nchans // 2])
    op = O.subband_plan(freq, n, 0.0, hi, fs, fe, step, ds, sb_width=width)
    d1, r2 = plan.tables()
    return plan, x, O.subband_sums(ref, nchans, op, d1, r2)


@pytest.mark.parametrize("n,nchans,nbits,hi,step,ds,width,band,zdm,iqrm", [
    (2560, 64, 8, 100.0, 0.5, 1, 32, 0.0, False, False),     # one tile of every segment
    (2561, 64, 8, 100.0, 0.5, 1, 32, 0.0, False, False),
    (2527, 64, 8, 500.0, 0.5, 1, 16, 0.0, True, True),
    (5, 64, 8, 20.0, 0.5, 1, 32, 0.0, False, False),         # fewer columns than segments
    (37, 64, 16, 20.0, 0.5, 1, 32, 0.0, False, False),
    (10243, 97, 8, 260.0, 0.5, 1, 33, 0.1, True, True),      # channels off the load words
    (4099, 130, 16, 260.0, 0.5, 1, 64, 0.1, True, True),
    (4096, 256, 8, 100.0, 0.3, 1, 64, 0.0, False, True),
    (3001, 260, 8, 100.0, 0.3, 1, 65, 0.0, False, False),    # 32-bit subband sums
    (3000, 384, 8, 60.0, 0.3, 1, 128, 0.0, True, False),
    (3000, 400, 8, 60.0, 0.3, 1, 129, 0.0, False, False),    # fields moved out inside a subband
    (2900, 600, 8, 60.0, 0.3, 1, 300, 0.0, False, False),
    (2900, 320, 16, 60.0, 0.3, 1, 160, 0.0, False, False),
    (9001, 128, 8, 300.0, 0.5, 2, 32, 0.2, True, True),      # binned
    (8003, 128, 16, 300.0, 0.5, 4, 32, 0.0, False, True),
    (3000, 64, 8, 3000.0, 200.0, 1, 32, 0.0, True, True),    # delays beyond the chunk, few rows
    (3000, 64, 16, 3000.0, 100.0, 1, 32, 0.0, False, False),
    (70000, 64, 8, 400.0, 2.0, 1, 16, 0.0, False, False),    # several tiles
])
@pytest.mark.parametrize("full", [False, True])
def test_subband_equals_oracle(n, nchans, nbits, hi, step, ds, width, band, zdm, iqrm, full):
    plan, x, want = subband(n, nchans, nbits, hi, step, ds, width, band, zdm, iqrm, full=full)
    out = to_np(plan.run(dev(x)))
    assert out.shape == want.shape and np.array_equal(out, want)
    host = plan.run_host(x)
    assert np.array_equal(host, want)


@pytest.mark.parametrize("n,nc,nbits,hi,step", [
    (2560, 65, 8, 100.0, 0.5), (2561, 129, 8, 300.0, 1.0), (2559, 258, 8, 64.0, 4.0),
    (1000, 300, 16, 100.0, 0.5), (1283, 33, 16, 15.0, 1.0), (9, 130, 8, 20.0, 1.0),
    (700, 64, 8, 3000.0, 300.0),
])
def test_brute_force_equals_oracle(n, nc, nbits, hi, step):
    x = data(n, nc, nbits, full=True)
    tsamp, foff = 1e-4, 300.0 / nc
    freq = O.freq_table_fil(1150.0, foff, nc)
    fs, fe = float(F32(freq[0])), float(F32(freq[-1]))
    hdr = dict(tsamp=tsamp, fch1=1150.0, foff=foff, nbits=nbits, nchans=nc, ndata=n)
    ts = n * tsamp * 0.49
    plan = Plan(hdr, 0.0, hi, fs, fe, step, 1, ts, algorithm="brute", freq_mode="fil")
    want = np.concatenate(O.bruteforce_cpu(x, nc, freq, tsamp, 0.0, hi, fs, fe, step, 1, ts,
                                           delay=plan.tables()[0]), axis=1)
    assert np.array_equal(to_np(plan.run(dev(x))), want)


@pytest.mark.parametrize("n,nc,nbits,hi,step,ds,frac", [
    (6001, 65, 8, 100.0, 1.0, 2, 0.1667), (5121, 130, 8, 300.0, 2.0, 3, 0.21),
    (5120, 64, 8, 300.0, 1.0, 2, 0.25), (4000, 33, 16, 200.0, 1.0, 4, 0.3),
    (4001, 130, 16, 200.0, 5.0, 2, 0.49), (9001, 40, 8, 100.0, 3.0, 8, 0.5),
    (6000, 40, 8, 100.0, 3.0, 16, 0.4), (6000, 40, 8, 100.0, 3.0, 17, 0.4),
])
def test_downsampled_brute_force_equals_oracle(n, nc, nbits, hi, step, ds, frac):
    x = data(n, nc, nbits, full=True)
    tsamp, foff = 1e-4, 300.0 / nc
    freq = O.freq_table_fil(1150.0, foff, nc)
    fs, fe = float(F32(freq[0])), float(F32(freq[-1]))
    hdr = dict(tsamp=tsamp, fch1=1150.0, foff=foff, nbits=nbits, nchans=nc, ndata=n)
    ts = n * tsamp * frac
    plan = Plan(hdr, 0.0, hi, fs, fe, step, ds, ts, algorithm="brute", freq_mode="fil")
    want = np.concatenate(O.bruteforce_cpu(x, nc, freq, tsamp, 0.0, hi, fs, fe, step, ds, ts,
                                           delay=plan.tables()[0]), axis=1)
    assert np.array_equal(to_np(plan.run(dev(x))), want)


@pytest.mark.parametrize("persistent", [False, True])
def test_batch_of_all_layouts_equals_oracle(persistent):
    specs = [(3001, 260, 8, 100.0, 0.3, 1, 65, 0.0, False, False),
             (2561, 64, 8, 100.0, 0.5, 1, 32, 0.0, True, True),
             (3000, 64, 8, 3000.0, 200.0, 1, 32, 0.0, False, False),
             (4099, 130, 16, 260.0, 0.5, 1, 64, 0.1, False, False)]
    got = [subband(*s) for s in specs]
    batch = Batch([g[0] for g in got], persistent=persistent)
    outs = batch.run([dev(g[1]) for g in got])
    batch.status()
    for o, (_, _, want) in zip(outs, got):
        assert np.array_equal(to_np(o), want)


@pytest.mark.parametrize("n,nchans,hi,step,ds,width", [
    (511, 37, 100.0, 0.5, 1, 16), (513, 64, 300.0, 0.5, 1, 9), (2049, 130, 60.0, 0.3, 1, 64),
    (1027, 64, 3000.0, 100.0, 1, 32), (3001, 40, 200.0, 1.0, 2, 8), (70001, 16, 100.0, 4.0, 1, 8),
])
def test_32bit_sums_equal_oracle(n, nchans, hi, step, ds, width):
    rng = np.random.default_rng(n)
    x = rng.integers(0, 2 ** 32, size=(n, nchans), dtype=np.uint64).astype(np.uint32)
    x[rng.random(x.shape) < 0.9] = 2 ** 32 - 1
    xd = torch.from_numpy(x.view(np.int32)).cuda().view(torch.uint32)
    foff = float(F32(300.0 / nchans))
    hdr = dict(tsamp=float(F32(64e-6)), fch1=1150.0, foff=foff, nbits=32, nchans=nchans, ndata=n)
    freq = O.freq_table_header(hdr["fch1"], hdr["foff"], nchans)
    fs, fe = float(F32(freq[0])), float(F32(freq[-1]))
    plan = Plan(hdr, 0.0, hi, fs, fe, step, ds, algorithm="subband", subband_width=width)
    ref = O.time_binning(x.copy(), nchans, ds) if ds > 1 else x
    op = O.subband_plan(freq, n, 0.0, hi, fs, fe, step, ds, sb_width=width)
    want = O.subband_sums(ref, nchans, op, *plan.tables())
    got = plan.run(xd).view(torch.int64).cpu().numpy().view(np.uint64)
    assert np.array_equal(got, want)
    if ds > 1:
        return
    filfreq = O.freq_table_fil(1150.0, 300.0 / nchans, nchans)
    bs, be = float(F32(filfreq[0])), float(F32(filfreq[-1]))
    ts = n * 64e-6 * 0.49
    bp = Plan(dict(hdr, tsamp=64e-6, foff=300.0 / nchans), 0.0, hi, bs, be, step, 1, ts,
              algorithm="brute", freq_mode="fil")
    bw = np.concatenate(O.bruteforce_cpu(x, nchans, filfreq, 64e-6, 0.0, hi, bs, be, step, 1, ts,
                                         delay=bp.tables()[0]), axis=1)
    assert np.array_equal(bp.run(xd).view(torch.int64).cpu().numpy().view(np.uint64), bw)


# 32-bit layout by words: masks that change inside a tile of 64 samples, zero-DM offsets and
# zeroed channels, at tile remainders; rows of 37 channels do not start on a word.
@pytest.mark.parametrize("n,nchans,width", [(511, 36, 16), (2049, 132, 64), (3001, 40, 8), (1027, 37, 9)])
def test_32bit_layout_with_masks(n, nchans, width):
    rng = np.random.default_rng(n + nchans)
    x = rng.integers(0, 2 ** 32, size=(n, nchans), dtype=np.uint64).astype(np.uint32)
    foff = float(F32(300.0 / nchans))
    hdr = dict(tsamp=float(F32(64e-6)), fch1=1150.0, foff=foff, nbits=32, nchans=nchans, ndata=n)
    freq = O.freq_table_header(hdr["fch1"], hdr["foff"], nchans)
    fs, fe = float(F32(freq[0])), float(F32(freq[-1]))
    iq = IqrmParams(mode=0, radius_frac=0.1, nsigma=3.0, win_sec=n * 64e-6 * 0.4, hop_sec=n * 64e-6 * 0.2)
    plan = Plan(hdr, 0.0, 60.0, fs, fe, 0.5, 1, algorithm="subband", subband_width=width,
                zero_dm_mode="range", rfi=RfiParams(use_zero_dm=True, use_iqrm=True, iqrm=iq, use_mask=True),
                bad_channels=[2])
    ref = x.copy()
    cs, ce = plan.info["chan_start"], plan.info["chan_end"]
    t0, t1, masks = O.iqrm_masks(ref, nchans, cs, ce, float(F32(F32(64e-6) * F32(1))), iq)
    O.apply_window_masks(ref, nchans, t0, t1, masks)
    O.zero_dm_range_exact(ref, nchans, cs, ce)
    O.mark_channels(ref, nchans, [2])
    op = O.subband_plan(freq, n, 0.0, 60.0, fs, fe, 0.5, 1, sb_width=width)
    want = O.subband_sums(ref, nchans, op, *plan.tables())
    got = plan.run(torch.from_numpy(x.view(np.int32)).cuda().view(torch.uint32))
    assert np.array_equal(got.view(torch.int64).cpu().numpy().view(np.uint64), want)


# The layout leaves out the positions past each 64 channels' largest delay: several groups of
# channels, a band that starts inside one and off the load words, two chunks in turn.
@pytest.mark.parametrize("n,nchans,nbits,hi,band", [
    (6001, 390, 8, 150.0, 0.13), (6001, 388, 8, 900.0, 0.13), (9000, 260, 16, 150.0, 0.31),
    (4100, 516, 16, 900.0, 0.07),
])
def test_layout_up_to_the_largest_delays(n, nchans, nbits, hi, band):
    plan, x, want = subband(n, nchans, nbits, hi, 1.0, 1, 64, band, True, False)
    other = dev(np.ascontiguousarray(x[::-1]))
    plan.run(other)
    assert np.array_equal(to_np(plan.run(dev(x))), want)


# Zero-DM offsets by words: more and fewer words than the loads in flight, a band that starts
# and ends inside a word, masked segments.
@pytest.mark.parametrize("n,nchans,nbits,band", [
    (700, 1024, 8, 0.0), (701, 1028, 8, 0.13), (650, 2052, 8, 0.0007), (700, 36, 8, 0.1),
    (650, 512, 16, 0.0), (651, 518, 16, 0.13), (640, 30, 16, 0.1),
])
def test_zero_dm_by_words(n, nchans, nbits, band):
    plan, x, want = subband(n, nchans, nbits, 20.0, 1.0, 1, 64, band, True, True)
    assert np.array_equal(to_np(plan.run(dev(x))), want)


# Rows that start off a load word: binning by pairs and single channels, the layout's last
# channels, masks and offsets beside them; a tile's remainders in time.
@pytest.mark.parametrize("n,nchans,nbits,ds", [
    (2561, 97, 8, 1), (4100, 98, 8, 2), (4099, 99, 8, 4), (1030, 66, 8, 3), (8200, 65, 8, 8),
    (2050, 131, 16, 1), (2051, 130, 16, 2), (4103, 67, 16, 4),
])
def test_ragged_rows(n, nchans, nbits, ds):
    plan, x, want = subband(n, nchans, nbits, 60.0, 0.5, ds, 16, 0.1, True, True)
    assert np.array_equal(to_np(plan.run(dev(x))), want)


@pytest.mark.parametrize("n,nchans,width", [(513, 37, 9), (2049, 131, 64)])
def test_ragged_rows_of_32_bits(n, nchans, width):
    test_32bit_layout_with_masks(n, nchans, width)


# The same on whole tiles (launches of at least four blocks per SM; the cases above take half
# tiles): one tile of every segment, a sample less and more, a last segment of a few columns,
# odd channel counts, subbands wider than the packing holds, full-scale samples.
@pytest.mark.parametrize("n,nchans,nbits,hi,step,width", [
    (2560, 64, 8, 60.0, 0.01, 2), (2561, 64, 8, 60.0, 0.01, 2), (2559, 67, 8, 60.0, 0.01, 2),
    (5125, 33, 8, 60.0, 0.01, 2), (17921, 260, 8, 60.0, 0.005, 65), (17923, 129, 8, 60.0, 0.005, 129),
    (1280, 64, 16, 60.0, 0.01, 2), (1281, 67, 16, 60.0, 0.01, 2), (2561, 64, 16, 60.0, 0.01, 2),
])
def test_subband_on_whole_tiles(n, nchans, nbits, hi, step, width):
    plan, x, want = subband(n, nchans, nbits, hi, step, 1, width, 0.0, False, False, full=True)
    assert np.array_equal(to_np(plan.run(dev(x))), want)


@pytest.mark.parametrize("n,nc,nbits,trials", [
    (2560, 65, 8, 9490), (2561, 33, 8, 4800), (5119, 130, 8, 4790), (1280, 64, 16, 9490), (1281, 65, 16, 4800),
])
def test_brute_force_on_whole_tiles(n, nc, nbits, trials):
    x = data(n, nc, nbits, full=True)
    tsamp, foff, step = 1e-4, 300.0 / nc, 0.005
    freq = O.freq_table_fil(1150.0, foff, nc)
    fs, fe = float(F32(freq[0])), float(F32(freq[-1]))
    hdr = dict(tsamp=tsamp, fch1=1150.0, foff=foff, nbits=nbits, nchans=nc, ndata=n)
    hi, ts = (trials - 0.5) * step, n * tsamp * 0.49
    plan = Plan(hdr, 0.0, hi, fs, fe, step, 1, ts, algorithm="brute", freq_mode="fil")
    assert plan.out_shape[0] == trials
    want = np.concatenate(O.bruteforce_cpu(x, nc, freq, tsamp, 0.0, hi, fs, fe, step, 1, ts,
                                           delay=plan.tables()[0]), axis=1)
    assert np.array_equal(to_np(plan.run(dev(x))), want)


# A chunk whose subband sums fit the budget is summed as one time tile (each tile costs stage
# 1 the stage-2 halo and the skew of its rows again); the host path splits it to copy the
# first half out meanwhile.
@pytest.mark.parametrize("spec", [(70001, 64, 8, 400.0, 2.0, 1, 16, 0.0, False, False),
                                  (66000, 48, 16, 3000.0, 100.0, 1, 16, 0.0, False, False)])
def test_one_time_tile_where_the_sums_fit(spec):
    plan, x, want = subband(*spec)
    xd = dev(x)
    assert plan.run_profiled(xd)["stage1_launches"] == 1
    assert np.array_equal(to_np(plan.run(xd)), want)
    outs = [np.empty(want.shape, np.uint32) for _ in range(3)]
    for i in range(3):
        plan.run_host_async(x, outs[i])
        if i == 1:
            assert np.array_equal(to_np(plan.run(xd)), want)
    plan.run_host_join(sync=True)
    for o in outs:
        assert np.array_equal(o, want)


# Bins per block: chunks of few bins and channels take fewer, down to those loaded together.
@pytest.mark.parametrize("n,nchans,nbits,ds", [
    (400, 16, 8, 2), (415, 17, 8, 16), (9000, 41, 8, 16), (2600, 64, 8, 5), (333, 16, 16, 8), (40000, 33, 16, 3),
])
def test_binning_of_small_chunks(n, nchans, nbits, ds):
    plan, x, want = subband(n, nchans, nbits, 20.0, 0.5, ds, 16, 0.0, False, False)
    assert np.array_equal(to_np(plan.run(dev(x))), want)


# All phase rows of a downsampled brute-force chunk are laid out by one launch, also where the
# last phases have a sample less or none.
@pytest.mark.parametrize("n,nc,nbits,ds,frac", [
    (494, 26, 16, 16, 0.49), (1000, 65, 8, 7, 0.5), (4099, 64, 8, 2, 0.49), (2050, 66, 16, 3, 0.3), (13, 12, 8, 16, 0.9),
])
def test_one_launch_lays_out_all_phases(n, nc, nbits, ds, frac):
    x = data(n, nc, nbits)
    tsamp, foff = 1e-4, 300.0 / nc
    freq = O.freq_table_fil(1150.0, foff, nc)
    fs, fe = float(F32(freq[0])), float(F32(freq[-1]))
    hdr = dict(tsamp=tsamp, fch1=1150.0, foff=foff, nbits=nbits, nchans=nc, ndata=n)
    ts = n * tsamp * frac
    plan = Plan(hdr, 0.0, 8.0, fs, fe, 1.0, ds, ts, algorithm="brute", freq_mode="fil")
    want = np.concatenate(O.bruteforce_cpu(x, nc, freq, tsamp, 0.0, 8.0, fs, fe, 1.0, ds, ts,
                                           delay=plan.tables()[0]), axis=1)
    xd = dev(x)
    # the layout, and the sums of all slices or (windows too wide to stage) of each
    assert plan.run_profiled(xd)["launches"] <= 1 + -(-n // max(1, int(ts / tsamp)))
    assert np.array_equal(to_np(plan.run(xd)), want)
