"""A beam pushed often enough that its tail moves to the front of the stream's buffer
several times: the pushes together equal the plain call on the whole beam.  Chunks
shorter and longer than the tail, and channel counts off the load words (pushes then
start at unaligned addresses)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from astroflow_b200.dedisp import IqrmParams, Plan, RfiParams, Stream  # noqa: E402

F32 = np.float32


@pytest.mark.parametrize("nchans,nbits,chunk,dm_high", [
    (64, 8, 700, 20.0), (64, 8, 700, 0.5), (37, 8, 333, 10.0), (50, 16, 512, 20.0),
])
def test_many_pushes_equal_plain_call(nchans, nbits, chunk, dm_high):
    k = 13
    rng = np.random.default_rng(nchans + chunk)
    x = rng.integers(0, 2 ** nbits, size=(k * chunk, nchans)).astype(np.uint8 if nbits == 8 else np.uint16)
    foff = float(F32(300.0 / nchans))
    hdr = dict(tsamp=float(F32(64e-6)), fch1=1150.0, foff=foff, nbits=nbits, nchans=nchans, ndata=chunk)
    fe = float(F32(np.float64(F32(1150.0)) + np.float64(F32(foff)) * (nchans - 1)))
    to_dev = lambda a: (torch.from_numpy(a.view(np.int16)).cuda().view(torch.uint16)  # noqa: E731
                        if nbits == 16 else torch.from_numpy(a).cuda())
    s = Stream(hdr, 0.0, dm_high, 1150.0, fe, 0.5, subband_width=16)
    tail = s.info["tail_samples"]
    assert (2 * (tail + chunk) - tail) // chunk < k  # the buffer's end is reached
    outs = [s.push(to_dev(x[i * chunk:(i + 1) * chunk])).view(torch.int32).cpu().numpy() for i in range(k)]
    padded = np.concatenate([np.zeros((tail, nchans), x.dtype), x])
    full = Plan(dict(hdr, ndata=padded.shape[0]), 0.0, dm_high, 1150.0, fe, 0.5, subband_width=16)
    want = full.run(to_dev(padded)).view(torch.int32).cpu().numpy()[:, :k * chunk]
    assert np.array_equal(np.concatenate(outs, axis=1), want)


def beam_and_windows(nchans, nbits, chunk, dm_high, k, seed, iqrm=True):
    """A stream with its RFI stages, k chunks of a beam, and what each push gives: the plain
    call on [tail | chunk]."""
    rng = np.random.default_rng(seed)
    x = rng.integers(0, 2 ** nbits // 4, size=(k * chunk, nchans)).astype(np.uint8 if nbits == 8 else np.uint16)
    for c in range(3, nchans, 11):  # channels that turn noisy for a while
        a = int(rng.integers(0, (k - 2) * chunk))
        x[a:a + 2 * chunk, c] = rng.integers(0, 2 ** nbits, 2 * chunk)
    foff = float(F32(300.0 / nchans))
    hdr = dict(tsamp=float(F32(64e-6)), fch1=1150.0, foff=foff, nbits=nbits, nchans=nchans, ndata=chunk)
    fe = float(F32(np.float64(F32(1150.0)) + np.float64(F32(foff)) * (nchans - 1)))
    kw = dict(subband_width=16, zero_dm_mode="range", bad_channels=[2],
              rfi=RfiParams(use_zero_dm=True, use_mask=True, use_iqrm=iqrm,
                            iqrm=IqrmParams(mode=1, radius_frac=0.1, nsigma=3.0,
                                            win_sec=chunk * 64e-6 * 0.6, hop_sec=chunk * 64e-6 * 0.3)))
    s = Stream(hdr, 0.0, dm_high, 1150.0, fe, 0.5, **kw)
    tail = s.info["tail_samples"]
    plan = Plan(dict(hdr, ndata=tail + chunk), 0.0, dm_high, 1150.0, fe, 0.5, **kw)
    padded = np.concatenate([np.zeros((tail, nchans), x.dtype), x])
    d = torch.from_numpy(padded.view(np.int16) if nbits == 16 else padded).cuda()
    d = d.view(torch.uint16) if nbits == 16 else d
    want = [plan.run(d[i * chunk:(i + 1) * chunk + tail].contiguous()).view(torch.int32).cpu().numpy()[:, :chunk]
            for i in range(k)]
    return s, [d[tail + i * chunk:tail + (i + 1) * chunk].contiguous() for i in range(k)], want


@pytest.mark.parametrize("nchans,nbits,chunk,dm_high", [(64, 8, 700, 20.0), (64, 8, 700, 0.5), (50, 16, 512, 20.0),
                                                       (64, 8, 300, 80.0)])
def test_pushes_with_masks_across_the_tails_move(nchans, nbits, chunk, dm_high):
    s, chunks, want = beam_and_windows(nchans, nbits, chunk, dm_high, 13, 5)
    for c, w in zip(chunks, want):
        assert np.array_equal(s.push(c).view(torch.int32).cpu().numpy(), w)


# A graph of one or several pushes, replayed over a beam and mixed with plain pushes, wherever
# the tail is at its capture.
@pytest.mark.parametrize("pushes,before", [(1, 1), (1, 4), (2, 1), (2, 2), (3, 3)])
@pytest.mark.parametrize("nchans,nbits,chunk,dm_high", [(64, 8, 700, 20.0), (64, 8, 700, 0.5), (37, 8, 333, 10.0),
                                                       (64, 8, 300, 80.0)])
def test_captured_pushes_continue_the_beam(nchans, nbits, chunk, dm_high, pushes, before):
    s, chunks, want = beam_and_windows(nchans, nbits, chunk, dm_high, before + 3 * pushes + 5, 6, iqrm=nchans == 64)
    chunks, want = iter(chunks), iter(want)
    check = lambda out: np.array_equal(out.view(torch.int32).cpu().numpy(), next(want))  # noqa: E731
    for _ in range(before):
        assert check(s.push(next(chunks)))
    bufs = [(torch.empty(s.chunk_shape, dtype=torch.uint8, device="cuda"), s.empty_output()) for _ in range(pushes)]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        for c, o in bufs:
            s.push(c, o)
    for rounds in (2, 1):
        for _ in range(rounds):
            for c, _ in bufs:
                c.copy_(next(chunks))
            graph.replay()
            for _, o in bufs:
                assert check(o)
        if rounds == 2:
            torch.cuda.synchronize()
    for _ in range(5):
        assert check(s.push(next(chunks)))
    del graph
