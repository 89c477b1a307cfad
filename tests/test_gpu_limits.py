"""Calls at the limits of a launch, a row or the device: more slices than a grid dimension
holds, rows of more than 2^31 samples, staged windows as wide as shared memory, trial steps so
coarse that rows are staged by eight or not at all, plans whose folded layout does not fit."""
import os
import subprocess
import sys

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from test_gpu_fold import dev, subband, to_np  # noqa: E402


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


# Trial steps around the limits of sixteen and eight rows a block, and past both: 8 bits about
# 10.4 and 22.5, 16 bits 5.5 and 11.  Batches launch the staged sums together; plans on the
# direct kernels run on their own.
@pytest.mark.parametrize("nbits,step,staged", [(8, 13.0, True), (8, 22.0, True), (8, 22.6, False),
                                               (16, 5.7, True), (16, 10.9, True), (16, 11.3, False)])
def test_brute_force_with_coarse_steps(nbits, step, staged):
    from astroflow_b200.dedisp import Batch, Plan
    from oracle import oracle as O

    n, nc, tsamp = 100003, 16, 82e-6
    x = np.random.default_rng(4).integers(0, 2 ** nbits, (n, nc)).astype(np.uint8 if nbits == 8 else np.uint16)
    freq = O.freq_table_fil(400.0, 25.0, nc)
    fs, fe = float(np.float32(freq[0])), float(np.float32(freq[-1]))
    hdr = dict(tsamp=tsamp, fch1=400.0, foff=25.0, nbits=nbits, nchans=nc, ndata=n)
    ts = n * tsamp * 0.49
    plan = Plan(hdr, 0.0, 26.5 * step, fs, fe, step, 1, ts, algorithm="brute", freq_mode="fil")
    want = np.concatenate(O.bruteforce_cpu(x, nc, freq, tsamp, 0.0, 26.5 * step, fs, fe, step, 1, ts,
                                           delay=plan.tables()[0]), axis=1)
    assert np.array_equal(to_np(plan.run(dev(x))), want)
    for persistent in (False, True):
        batch = Batch([plan], persistent=persistent)
        assert np.array_equal(to_np(batch.run([dev(x)])[0]), want)
        batch.status()
        assert persistent or batch.info["own_plans"] == (0 if staged else 1)


# The same for the two stages: wide rows of stage 2 (the twin's, 32-bit sums') and, with one
# subband, of stage 1 (16-bit and 32-bit sums), up to steps that no staged form takes.
@pytest.mark.parametrize("n,nchans,nbits,trials,step,width,staged", [
    (30011, 64, 8, 99, 10.0, 16, True), (50001, 64, 8, 70, 30.0, 16, True), (50001, 64, 8, 70, 40.0, 16, True),
    (30011, 64, 16, 99, 10.0, 16, True), (90001, 32, 16, 70, 40.0, 16, False), (90001, 32, 16, 70, 75.0, 16, False),
    (40003, 64, 16, 99, 20.0, 16, True),
    (30011, 256, 8, 99, 10.0, 128, True), (60002, 48, 8, 331, 8.0, 64, True), (60002, 48, 8, 331, 9.5, 64, False),
    (60002, 70, 8, 331, 8.0, 70, True), (60002, 48, 16, 331, 4.0, 48, True), (60002, 48, 16, 331, 5.0, 48, False),
])
def test_subbands_with_coarse_steps(n, nchans, nbits, trials, step, width, staged):
    from astroflow_b200.dedisp import Batch

    plan, x, want = subband(n, nchans, nbits, step * (trials - 0.5), step, 1, width, 0.0, False, False, full=True)
    assert np.array_equal(to_np(plan.run(dev(x))), want)
    assert np.array_equal(plan.run_host(x), want)
    for persistent in (False, True):
        batch = Batch([plan], persistent=persistent)
        assert np.array_equal(to_np(batch.run([dev(x)])[0]), want)
        batch.status()
        assert persistent or batch.info["own_plans"] == (0 if staged else 1)


def test_folded_subband_sums_stay_near_their_budget():
    """16,001 trials over 4096 channels hold 513 KB of subband sums per word of a time tile:
    the tiles' padding must not add up to gigabytes (budget 2 GiB, layout 0.9 GB)."""
    from astroflow_b200.dedisp import Plan

    n, nc, f32 = 1 << 17, 4096, np.float32
    foff = float(f32(500.0 / nc))
    hdr = dict(tsamp=float(f32(4.9e-5)), fch1=1000.0, foff=foff, nbits=8, nchans=nc, ndata=n)
    plan = Plan(hdr, 0.0, 400.0, 1000.0, float(f32(1000.0) + f32(nc - 1) * f32(foff)), 0.025, 1)
    assert plan.out_shape[0] == 16001 and plan.info["subband_sum_copies"] == 1
    assert plan.info["workspace_bytes"] < 3.8e9
    plan.close()


def test_folded_brute_force_holds_a_segment_and_the_largest_delay():
    """Words of the folded layout end at the largest delay past a segment: a quarter of the
    chunk and 34,000 samples of delay per channel, where the rows in time order need the
    chunk, the delay and a slice."""
    from astroflow_b200.dedisp import Plan
    from oracle import oracle as O

    n, nc, tsamp = 1 << 17, 64, 6.4e-5
    freq = O.freq_table_fil(1000.0, 500.0 / nc, nc)
    fs, fe = float(np.float32(freq[0])), float(np.float32(freq[-1]))
    hdr = dict(tsamp=tsamp, fch1=1000.0, foff=500.0 / nc, nbits=8, nchans=nc, ndata=n)
    plan = Plan(hdr, 0.0, 950.0, fs, fe, 1.0, 1, n * tsamp * 0.49, algorithm="brute", freq_mode="fil")
    most = int(plan.tables()[0].max())
    assert 30000 < most < 40000
    assert plan.info["workspace_bytes"] < nc * 4 * (n // 4 + most + 4096) + plan.out_shape[0] * nc * 8 + (1 << 16)
    # delays twice as long as the plan's own: the rows grow with them
    x = np.random.default_rng(8).integers(0, 256, (n, nc)).astype(np.uint8)
    table = np.minimum(plan.tables()[0] * 2, most + 15000).astype(np.int32)
    plan.set_delay_table(table)
    want = np.concatenate(O.bruteforce_cpu(x, nc, freq, tsamp, 0.0, 950.0, fs, fe, 1.0, 1, n * tsamp * 0.49,
                                           delay=table), axis=1)
    assert np.array_equal(to_np(plan.run(dev(x))), want)
    plan.close()


def test_runs_beside_the_legacy_stream_after_a_new_delay_table():
    """A table whose delays change the layout's size takes new buffers; a run on a stream that
    does not wait for the legacy one follows at once."""
    from astroflow_b200.dedisp import Plan
    from oracle import oracle as O

    n, nc, tsamp = 20000, 300, 6.4e-5
    freq = O.freq_table_fil(1000.0, 500.0 / nc, nc)
    fs, fe = float(np.float32(freq[0])), float(np.float32(freq[-1]))
    hdr = dict(tsamp=tsamp, fch1=1000.0, foff=500.0 / nc, nbits=8, nchans=nc, ndata=n)
    plan = Plan(hdr, 0.0, 99.5, fs, fe, 1.0, 1, n * tsamp * 0.49, algorithm="brute", freq_mode="fil")
    x = np.random.default_rng(9).integers(0, 256, (n, nc)).astype(np.uint8)
    xd, out, own = dev(x), plan.empty_output(), plan.tables()[0]
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for k in (3, 0, 2, 1):
        table = (own * k // 3).astype(np.int32)
        plan.set_delay_table(table)
        plan.run(xd, out, side)
        side.synchronize()
        want = np.concatenate(O.bruteforce_cpu(x, nc, freq, tsamp, 0.0, 99.5, fs, fe, 1.0, 1, n * tsamp * 0.49,
                                               delay=table), axis=1)
        assert np.array_equal(to_np(out), want)


# A folded chunk takes up to four times its bytes: with less memory left than that, the plan
# keeps the chunk in time order (subband sums: shorter time tiles come first).  In a process
# of its own, whose memory holds nothing else; MiB left for the plan or the stream (time order /
# folded take 480 / 658, 1143 / 1452 and, with the stream's own buffer, 2191 / 2409).
# "host" has the plan and lacks memory for its host path's own buffers (577 MiB).
SHORT_OF_MEMORY = """
import sys
import numpy as np
import torch
from astroflow_b200.dedisp import Plan, Stream

kind, nbits, leave = sys.argv[1], int(sys.argv[2]), int(sys.argv[3]) << 20
n, nc, f32 = 1 << (17 if kind == "stream" else 18), 1024, np.float32
x = torch.randint(0, 127, (n, nc * nbits // 8), dtype=torch.uint8, device="cuda").view(
    torch.uint8 if nbits == 8 else torch.uint16)
hdr = dict(tsamp=float(f32(1.6e-4)), fch1=400.0, foff=float(f32(400.0 / nc)), nbits=nbits, nchans=nc, ndata=n)
fe = float(f32(400.0) + f32(nc - 1) * f32(400.0 / nc))

def make():
    if kind in ("brute", "host"):
        return Plan(hdr, 0.0, 800.0, 400.0, fe, 2.5, 1, n * 1.6e-4 * 0.49, algorithm="brute", freq_mode="fil")
    if kind == "subband":
        return Plan(hdr, 0.0, 600.0, 400.0, fe, 1.0, 1)
    return Stream(hdr, 0.0, 800.0, 400.0, fe, 0.5, 1)

def run(p):
    p.push(x, out) if kind == "stream" else p.run(x, out)
    return out.view(torch.int32).cpu()

p = make()
out = p.empty_output()
want = run(p)
folded = p.info["workspace_bytes"]
p.close()
out.view(torch.int32).zero_()
torch.cuda.synchronize()
torch.cuda.empty_cache()
if kind == "host":
    p = make()
    host = x.cpu().numpy()
    del out
    torch.cuda.empty_cache()
hog = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
if kind == "host":
    for _ in range(2):
        assert np.array_equal(p.run_host(host).view(np.int32), want.numpy())
else:
    p = make()
    assert p.info["workspace_bytes"] < folded, (p.info["workspace_bytes"], folded)
    assert torch.equal(run(p), want)
"""


@pytest.mark.parametrize("kind,nbits,leave_mb", [("brute", 8, 630), ("subband", 16, 1300), ("subband", 16, 800),
                                                 ("stream", 16, 2310), ("host", 8, 500)])
def test_plans_whose_folded_layout_does_not_fit(kind, nbits, leave_mb):
    torch.cuda.empty_cache()
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", SHORT_OF_MEMORY, kind, str(nbits), str(leave_mb)], cwd=root,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
