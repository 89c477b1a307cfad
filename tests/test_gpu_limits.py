"""Calls at the limits of a launch, a row or the device: more slices than a grid dimension
holds, rows of more than 2^31 samples, staged windows as wide as shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_more_slices_than_a_launch_takes():
    """Slices too wide for the two-pass resize, more of them than a grid's y dimension: the
    ones past 65,535 too are resized and colored."""
    pytest.importorskip("cv2")
    from astroflow_b200 import postprocess
    from oracle import cv2_images as CVI

    target, width, n = 8, 2000, 70000
    raw = np.random.default_rng(7).integers(0, 1 << 20, (1, width + 16)).astype(np.uint32)
    d = torch.from_numpy(raw.view(np.int32)).cuda().view(torch.uint32)
    starts = np.arange(n) % 7
    got = postprocess.device_images(d, starts, np.full(n, width), target=target).cpu().numpy()
    want = np.stack([CVI.image(raw[:, s:s + width], target) for s in range(7)])
    assert np.array_equal(got, want[starts])


def test_rows_past_two_to_the_31():
    """One trial (DM 0) over two channels of 32-bit samples longer than 2^31: the layout and
    the sums reach the end of the rows (about 52 GB on the device)."""
    from astroflow_b200.dedisp import Plan

    n = 2 ** 31 + 4099
    if torch.cuda.mem_get_info()[0] < 60e9:
        pytest.skip("needs 60 GB of device memory")
    x = torch.empty((n, 2), dtype=torch.int32, device="cuda").random_(0, 2 ** 31 - 1)
    hdr = dict(tsamp=6.4e-5, fch1=1150.0, foff=1.0, nbits=32, nchans=2, ndata=n)
    plan = Plan(hdr, 0.0, 0.0, 1150.0, 1151.0, 1.0, 1)
    out = plan.run(x.view(torch.uint32)).view(torch.int64)
    assert out.shape == (1, n)
    for a in list(range(0, n, n // 5)) + [2 ** 31 - (1 << 20), 2 ** 31 - 70, n - 5000]:
        b = min(n, a + (1 << 20))
        assert torch.equal(out[0, a:b], x[a:b].to(torch.int64).sum(1)), a


# The windows of sixteen 8-bit rows around what a block's shared memory holds beside the
# slices through which the sums leave (36 KB): the spread of the rows' delays in samples.
@pytest.mark.parametrize("step,spread", [(10.2, 35493), (10.4, 36189), (10.7, 37233), (11.0, 38277),
                                         (11.2, 38973)])
def test_brute_force_windows_at_the_shared_memory_limit(step, spread):
    from astroflow_b200.dedisp import Plan
    from oracle import oracle as O

    n, nc, tsamp = 50001, 16, 82e-6
    x = np.random.default_rng(3).integers(0, 256, (n, nc)).astype(np.uint8)
    freq = O.freq_table_fil(400.0, 25.0, nc)
    fs, fe = float(np.float32(freq[0])), float(np.float32(freq[-1]))
    hdr = dict(tsamp=tsamp, fch1=400.0, foff=25.0, nbits=8, nchans=nc, ndata=n)
    ts = n * tsamp * 0.49
    plan = Plan(hdr, 0.0, 15.5 * step, fs, fe, step, 1, ts, algorithm="brute", freq_mode="fil")
    delay = plan.tables()[0]
    assert plan.out_shape[0] == 16 and abs(int((delay.max(0) - delay.min(0)).max()) - spread) < 30
    want = np.concatenate(O.bruteforce_cpu(x, nc, freq, tsamp, 0.0, 15.5 * step, fs, fe, step, 1, ts,
                                           delay=delay), axis=1)
    got = plan.run(torch.from_numpy(x).cuda()).view(torch.int32).cpu().numpy().view(np.uint32)
    assert np.array_equal(got, want)
