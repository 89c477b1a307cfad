"""A beam pushed often enough that its tail moves to the front of the stream's buffer
several times: the pushes together equal the plain call on the whole beam.  Chunks
shorter and longer than the tail, and channel counts off the load words (pushes then
start at unaligned addresses)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from astroflow_b200.dedisp import Plan, Stream  # noqa: E402

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
