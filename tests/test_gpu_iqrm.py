"""IQRM masks on the GPU against the oracle's restatement, bit for bit, where the
word-wise sums, the window runs and the order statistics can go wrong: bands of one to a
few thousand channels that start off a word, sample counts around the sixteen-row
blocks and the chunk length, overlapping windows, and flat bands whose differences tie."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
from astroflow_b200.dedisp import IqrmParams, iqrm_masks_noalloc  # noqa: E402
from oracle import oracle as O  # noqa: E402

TSAMP = 1e-3


def to_dev(x):
    signed = {1: np.uint8, 2: np.int16, 4: np.int32}[x.dtype.itemsize]
    t = torch.from_numpy(x.view(signed)).cuda()
    return t.view({1: torch.uint8, 2: torch.uint16, 4: torch.uint32}[x.dtype.itemsize])


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("nbits,nchans,cs,ce,nsamp,win,flat", [
    (8, 8, 0, 2, 17, 0.0, False),
    (8, 64, 3, 62, 1023, 0.3, False),
    (8, 512, 1, 510, 1025, 0.5, False),
    (8, 2048, 0, 2047, 4099, 1.0, False),
    (8, 258, 5, 257, 2500, 0.7, False),
    (8, 256, 0, 256, 1040, 0.4, True),
    (16, 130, 1, 129, 3001, 0.6, False),
    (16, 4097, 0, 4096, 515, 0.0, False),
    (32, 100, 7, 93, 1500, 0.25, False),
])
def test_masks_equal_oracle(nbits, nchans, cs, ce, nsamp, win, flat, mode):
    rng = np.random.default_rng(nchans * 7 + nsamp)
    dt = {8: np.uint8, 16: np.uint16, 32: np.uint32}[nbits]
    mid, sd = {8: (128, 20), 16: (32768, 2000), 32: (1e6, 6e4)}[nbits]
    x = rng.normal(mid, sd, (nsamp, nchans))
    if flat:  # whole blocks of channels equal: differences tie at zero
        x[:] = mid
        x[:, ::7] += rng.normal(0, sd, (nsamp, len(range(0, nchans, 7))))
    for c in rng.choice(nchans, max(1, nchans // 16), replace=False):
        x[:, c] += 4 * sd * np.sin(np.arange(nsamp) * 0.37) + 2 * sd
    x = np.clip(np.rint(x), 0, 2.0 ** nbits - 1).astype(dt)
    iq = IqrmParams(mode=mode, radius_frac=0.1, nsigma=3.0, geofactor=1.5, win_sec=win,
                    hop_sec=win / 2, include_tail=True)
    t0, t1, want = O.iqrm_masks(x.copy(), nchans, cs, ce, TSAMP, iq)
    masks = torch.full((len(t0) + 1, nchans), 9, dtype=torch.uint8, device="cuda")
    bounds = torch.zeros((len(t0) + 1, 2), dtype=torch.int32, device="cuda")
    n = iqrm_masks_noalloc(to_dev(x), nchans, cs, ce, TSAMP, iq, masks, bounds)
    assert n == len(t0)
    assert np.array_equal(masks[:n].cpu().numpy(), want)
    assert np.array_equal(bounds[:n].cpu().numpy(), np.stack([t0, t1], 1).astype(np.int32))


# Bands around the block sizes of the order statistics (one warp, four, sixteen).
@pytest.mark.parametrize("csub", [1, 2, 31, 32, 33, 127, 128, 129])
def test_masks_of_few_channels(csub):
    test_masks_equal_oracle(8, csub + 6, 3, 3 + csub, 700, 0.2, False, 1)


# Windows that start a few samples apart are summed one by one, the rest in shared runs.
@pytest.mark.parametrize("nbits,nchans,nsamp,win,hop", [
    (8, 240, 100, 32, 2), (8, 97, 100, 32, 3), (16, 60, 300, 7, 1), (16, 61, 128, 100, 9), (32, 30, 90, 30, 2),
    (8, 64, 2000, 200, 70), (16, 64, 2000, 200, 63),
])
def test_masks_of_many_short_windows(nbits, nchans, nsamp, win, hop):
    rng = np.random.default_rng(nsamp + nchans)
    x = rng.integers(0, 200, (nsamp, nchans)).astype({8: np.uint8, 16: np.uint16, 32: np.uint32}[nbits])
    x[:, 5] //= 9
    x[nsamp // 2:, 17] = 3
    iq = IqrmParams(mode=1, radius_frac=0.1, nsigma=3.0, geofactor=1.5, win_sec=win * TSAMP + 1e-7,
                    hop_sec=hop * TSAMP + 1e-7, include_tail=True)
    t0, t1, want = O.iqrm_masks(x.copy(), nchans, 2, nchans - 1, TSAMP, iq)
    masks = torch.full((len(t0), nchans), 9, dtype=torch.uint8, device="cuda")
    bounds = torch.zeros((len(t0), 2), dtype=torch.int32, device="cuda")
    assert iqrm_masks_noalloc(to_dev(x), nchans, 2, nchans - 1, TSAMP, iq, masks, bounds) == len(t0)
    assert t0[1] == hop and np.array_equal(masks.cpu().numpy(), want)


def test_widest_band():
    """The widest band whose differences a block holds, and one channel more."""
    test_masks_equal_oracle(8, 32769, 0, 32768, 20, 0.0, False, 1)
    x = torch.zeros((8, 32770), dtype=torch.uint8, device="cuda")
    masks = torch.zeros((1, 32770), dtype=torch.uint8, device="cuda")
    bounds = torch.zeros((1, 2), dtype=torch.int32, device="cuda")
    with pytest.raises(ValueError, match="at most 32768 channels"):
        iqrm_masks_noalloc(x, 32770, 0, 32769, TSAMP, IqrmParams(radius_frac=1e-4, win_sec=0.0), masks, bounds)
