"""What users of the library run: dedispersion plans, beams, batches, images and the drop-in call.

A case is a dict of plain values; `kind` says which public entry point it goes through:

  plan    Plan.run on a resident chunk (subband or brute force)
  stream  Stream.push of one chunk of a beam
  batch   Batch.run of several chunks of different geometry
  images  device_images on a resident DM-time plane
  dropin  _astroflow_core._dedisperse_spec on a host array, images back on the host

Inputs are seeded Gaussian noise in the sample type with sinusoidal RFI channels, broadband
impulses and dispersed pulses, as real chunks have them.  The outputs are whole numbers (DM-time
sums and image bytes), so there is nothing to give in 64-bit floating point.
"""
import math
import random

import numpy as np
import torch

KDM = 4148.808
TSAMP = 49.152e-6
IQRM = {
    # one window over the chunk, radius of five lags (of 4096 channels)
    "one_window": dict(mode=1, radius_frac=0.00134, nsigma=3.0, geofactor=1.5, win_sec=0.0,
                       hop_sec=0.5, include_tail=True),
    # the defaults: 5 s windows every 2.5 s, radius a tenth of the band
    "default": dict(mode=0, radius_frac=0.10, nsigma=3.0, geofactor=1.5, win_sec=5.0,
                    hop_sec=2.5, include_tail=True),
}


def _plan(name, nchans, nsamp, nbits, dm_low, dm_high, dm_step, *, algorithm="subband", width=64,
          ds=1, f_hi=1500.0, bandwidth=500.0, tsamp=TSAMP, zero_dm="none", iqrm="none",
          band_low=0.0, t_sample=0.5, kind="plan"):
    c = dict(kind=kind, nchans=nchans, nsamp=nsamp, nbits=nbits, dm_low=dm_low, dm_high=dm_high,
             dm_step=dm_step, algorithm=algorithm, width=width, ds=ds, f_hi=f_hi,
             bandwidth=bandwidth, tsamp=tsamp, zero_dm=zero_dm, iqrm=iqrm, band_low=band_low,
             t_sample=t_sample)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # a short search file of a 336-channel receiver (millisecond samples, 591 trials): the
        # smallest call, where launches and latency count
        _plan("file-336ch", 336, 5120, 8, 10.0, 600.0, 1.0, width=32, f_hi=1488.0,
              bandwidth=336.0, tsamp=1.2656e-3),
        # 6.4 s of 4096 channels over DM 0-3000 with both RFI stages: the usual search chunk
        _plan("chunk-4096ch", 4096, 1 << 17, 8, 0.0, 3000.0, 0.5, zero_dm="callsite",
              iqrm="one_window"),
        # the same search over 51.5 s at once: the largest call
        _plan("long-4096ch", 4096, 1 << 20, 8, 0.0, 3000.0, 0.5, zero_dm="callsite",
              iqrm="one_window"),
        # 16-bit samples of 8192 channels, fine DM steps
        _plan("u16-8192ch", 8192, 1 << 18, 16, 0.0, 500.0, 0.25, zero_dm="callsite",
              iqrm="one_window"),
        # a high-DM range on a ragged chunk: time binning, IQRM windows, range zero-DM
        _plan("binned-2048ch", 2048, 300001, 8, 500.0, 1500.0, 1.5, width=32, ds=4, f_hi=1550.0,
              bandwidth=300.0, zero_dm="range", iqrm="default"),
        # brute force over 1024 channels
        _plan("brute-1024ch", 1024, 1 << 17, 8, 0.0, 1000.0, 1.0, algorithm="brute"),
        # brute force with downsampling on odd sizes
        _plan("brute-ds2", 1000, 61441, 8, 0.0, 500.0, 1.0, algorithm="brute", ds=2),
        # 32-bit samples (sums of many beams or polarisations)
        _plan("u32-1024ch", 1024, 1 << 15, 32, 0.0, 500.0, 1.0, width=32),
        # one 0.5 s chunk of a real-time beam with its 7 s tail on the device
        _plan("beam-push", 4096, 10172, 8, 0.0, 3000.0, 1.0, zero_dm="callsite",
              iqrm="one_window", kind="stream"),
        # eight short chunks of different shape in one run
        dict(name="batch-8", kind="batch", nchunks=8, log2_low=15.0, log2_high=17.0, draw=11),
        # the detector's images of 12.9 s of a 3001-trial search, 0.5 s each
        dict(name="images-26", kind="images", rows=3001, cols=1 << 18, slice_cols=10172),
        # the pipeline's own call: host spectrum in, images out
        _plan("dropin-1024ch", 1024, 1 << 16, 8, 0.0, 500.0, 1.0, zero_dm="callsite",
              iqrm="default", kind="dropin"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["subband"] * 6 + ["brute"] * 2 + ["u32", "stream", "batch", "images", "dropin"])
    if kind == "images":
        cols = _log(rng, 2048, 1 << 18)
        return dict(kind="images", rows=rng.randint(200, 3001), cols=cols,
                    slice_cols=rng.randint(300, min(cols, 12000)))
    if kind == "batch":
        return dict(kind="batch", nchunks=rng.randint(2, 10), log2_low=13.0, log2_high=17.0,
                    draw=rng.randint(100, 10 ** 6))
    f_hi, bandwidth = rng.choice([(1500.0, 500.0), (1550.0, 300.0)])
    dm_high = rng.choice([300.0, 500.0, 1000.0, 1500.0, 3000.0])
    dm_step = rng.choice([0.5, 1.0, 1.5, 2.0])
    dm_low = rng.choice([0.0, 0.0, 10.0, 100.0])
    if kind == "brute":
        return _plan("", _log(rng, 128, 1024), _log(rng, 1 << 14, 1 << 17), rng.choice([8, 8, 16]),
                     dm_low, min(dm_high, 1000.0), dm_step * 2, algorithm="brute",
                     ds=rng.choice([1, 1, 1, 2]), f_hi=f_hi, bandwidth=bandwidth, t_sample=0.25)
    if kind == "u32":
        return _plan("", _log(rng, 128, 1024), _log(rng, 1 << 13, 1 << 15), 32, dm_low, 500.0,
                     dm_step * 2, width=32, f_hi=f_hi, bandwidth=bandwidth)
    if kind == "stream":
        return _plan("", 4 * _log(rng, 128, 1024), _log(rng, 2000, 20344), rng.choice([8, 8, 16]),
                     0.0, dm_high, max(dm_step, 1.0), f_hi=f_hi, bandwidth=bandwidth,
                     iqrm=rng.choice(["none", "one_window"]), kind="stream")
    if kind == "dropin":
        return _plan("", 4 * _log(rng, 64, 512), _log(rng, 1 << 15, 1 << 17), rng.choice([8, 16]),
                     dm_low, 500.0, 1.0, f_hi=f_hi, bandwidth=bandwidth, zero_dm="callsite",
                     iqrm=rng.choice(["none", "default"]), kind="dropin")
    nbits = rng.choice([8, 8, 8, 16])
    ds = rng.choice([1, 1, 1, 2, 4, 8])
    nchans = rng.choice([_log(rng, 256, 4096), 1024, 2048, 4096])
    return _plan("", nchans, _log(rng, 1 << 14, 1 << 19), nbits, dm_low, dm_high, dm_step,
                 width=rng.choice([16, 32, 32, 64, 64]), ds=ds, f_hi=f_hi, bandwidth=bandwidth,
                 zero_dm=rng.choice(["none", "callsite", "range"]),
                 iqrm=rng.choice(["none", "one_window", "default"]),
                 band_low=rng.choice([0.0, 0.0, 0.0, 0.1]))


# ---------------------------------------------------------------- inputs
_LEVEL = {8: (128.0, 20.0, 255.0), 16: (32768.0, 2000.0, 65535.0), 32: (1e6, 6e4, 4294967295.0)}
_TYPE = {8: torch.uint8, 16: torch.uint16, 32: torch.uint32}


def _chunk(nsamp, nchans, nbits, f_hi, bandwidth, tsamp, seed, dms=(120.0, 780.0)):
    """A seeded chunk [nsamp, nchans] on the GPU: noise, 5 % sinusoidal RFI channels, 20
    broadband impulses and one dispersed pulse per DM."""
    dev = torch.device("cuda")
    mean, sigma, vmax = _LEVEL[nbits]
    rng = np.random.default_rng(seed)
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    nr = max(1, nchans // 20)
    bad = torch.from_numpy(rng.choice(nchans, nr, replace=False)).to(dev)
    omega = torch.from_numpy(2 * np.pi / rng.integers(2, 201, nr)).float().to(dev)
    phase = torch.from_numpy(rng.uniform(0, 2 * np.pi, nr)).float().to(dev)
    hits = [(int(rng.integers(0, nsamp)), int(rng.integers(1, 5))) for _ in range(20)]
    freq = f_hi - (nchans - 1 - np.arange(nchans)) * (bandwidth / nchans)
    width = max(1e-3 / tsamp, 0.5)
    offs = torch.arange(-int(4 * width) - 1, int(4 * width) + 2, device=dev)
    shape = (0.6 * sigma * torch.exp(-0.5 * (offs / width) ** 2)).float()
    cols = torch.arange(nchans, device=dev)
    pulses = []
    for dm in dms:
        t0 = float(rng.uniform(0.05, 0.5)) * nsamp * tsamp
        at = np.rint((t0 + KDM * dm * (freq ** -2 - f_hi ** -2)) / tsamp).astype(np.int64)
        pulses.append(torch.from_numpy(at).to(dev))
    out = torch.empty((nsamp, nchans), dtype=_TYPE[nbits], device=dev)
    rows = max(1, (1 << 27) // nchans)
    for r0 in range(0, nsamp, rows):
        r1 = min(nsamp, r0 + rows)
        b = torch.randn((r1 - r0, nchans), generator=g, device=dev)
        b.mul_(sigma).add_(mean)
        t = torch.arange(r0, r1, device=dev, dtype=torch.float32)
        b[:, bad] += 3 * sigma * torch.sin(t[:, None] * omega + phase)
        for h, w in hits:
            if h < r1 and h + w > r0:
                b[max(h, r0) - r0:min(h + w, r1) - r0] += 2.5 * sigma
        for at in pulses:
            row = at[:, None] + offs
            ok = (row >= r0) & (row < r1)
            c = cols[:, None].expand_as(row)[ok]
            b.index_put_((row[ok] - r0, c), shape.expand_as(row)[ok], accumulate=True)
        b.round_().clamp_(0, vmax)
        out[r0:r1] = b.to(torch.int64 if nbits == 32 else torch.int32).to(_TYPE[nbits])
    return out


def _band(c):
    """Header fields and the band limits of the header's own float frequency table."""
    foff = np.float32(c["bandwidth"] / c["nchans"])
    fch1 = np.float32(c["f_hi"] - (c["nchans"] - 1) * (c["bandwidth"] / c["nchans"]))
    last = np.float32(np.float64(fch1) + np.float64(foff) * (c["nchans"] - 1))
    first = np.float32(fch1 + np.float32(c["band_low"]) * (last - fch1))
    hdr = dict(tsamp=float(np.float32(c["tsamp"])), fch1=float(fch1), foff=float(foff),
               nbits=c["nbits"], nchans=c["nchans"], ndata=c["nsamp"])
    return hdr, float(first), float(last)


def _rfi(c):
    from astroflow_b200.dedisp import IqrmParams, RfiParams

    q = IqrmParams(**IQRM[c["iqrm"]]) if c["iqrm"] != "none" else IqrmParams()
    return RfiParams(use_zero_dm=c["zero_dm"] != "none", use_iqrm=c["iqrm"] != "none", iqrm=q)


def _make_plan(c):
    from astroflow_b200.dedisp import Plan

    hdr, first, last = _band(c)
    more = dict(rfi=_rfi(c), zero_dm_mode="callsite" if c["zero_dm"] == "none" else c["zero_dm"])
    if c["algorithm"] == "brute":
        more = dict(freq_mode="fil")
    return Plan(hdr, c["dm_low"], c["dm_high"], first, last, c["dm_step"], c["ds"], c["t_sample"],
                algorithm=c["algorithm"], subband_width=c["width"], **more)


def _input(c, seed):
    return _chunk(c["nsamp"], c["nchans"], c["nbits"], c["f_hi"], c["bandwidth"], c["tsamp"], seed)


def _batch_cases(c):
    """The batch's chunks: nchan 1024-4096, 8 or 16 bits, two bands, DM up to 1500, downsampling 1-8."""
    rng = random.Random(c["draw"])
    got = []
    for _ in range(c["nchunks"]):
        f_hi, bandwidth = rng.choice([(1500.0, 500.0), (1550.0, 300.0)])
        got.append(_plan("", rng.choice([1024, 2048, 4096]),
                         int(2 ** rng.uniform(c["log2_low"], c["log2_high"])), rng.choice([8, 16]),
                         0.0, rng.choice([500.0, 1500.0]), rng.choice([0.5, 1.0, 1.5, 2.0]),
                         width=32, ds=rng.choice([1, 2, 4, 8]), f_hi=f_hi, bandwidth=bandwidth))
    return got


def prepare(case, seed):
    c = case
    if c["kind"] == "images":
        g = torch.Generator(device="cuda")
        g.manual_seed(seed)
        sums = torch.empty((c["rows"], c["cols"]), dtype=torch.uint32, device="cuda")
        for r in range(0, c["rows"], 256):
            n = min(256, c["rows"] - r)
            b = torch.randn((n, c["cols"]), generator=g, device="cuda") * 1280.0 + 524288.0
            sums[r:r + n] = b.round_().to(torch.int32).view(torch.uint32)
        starts = list(range(0, c["cols"], c["slice_cols"]))
        counts = [min(c["slice_cols"], c["cols"] - s) for s in starts]
        return dict(kind="images", sums=sums, starts=starts, counts=counts)
    if c["kind"] == "batch":
        from astroflow_b200.dedisp import Batch

        cases = _batch_cases(c)
        plans = [_make_plan(q) for q in cases]
        return dict(kind="batch", batch=Batch(plans), plans=plans,
                    xs=[_input(q, 100 * seed + i) for i, q in enumerate(cases)],
                    outs=[p.empty_output() for p in plans])
    if c["kind"] == "dropin":
        from astroflow_b200 import _astroflow_core as core

        hdr, first, last = _band(c)
        q = IQRM[c["iqrm"]] if c["iqrm"] != "none" else IQRM["default"]
        iqrm = core.IQRMconfig(q["mode"], q["radius_frac"], q["nsigma"], q["geofactor"],
                               q["win_sec"], q["hop_sec"], q["include_tail"])
        header = core.Header(0.0, hdr["tsamp"], hdr["fch1"], hdr["foff"], c["nbits"], c["nchans"],
                             c["nsamp"], "spectrum")
        cfg = core.RFIconfig(False, c["zero_dm"] != "none", c["iqrm"] != "none", iqrm)
        return dict(kind="dropin", data=_input(c, seed).cpu().numpy(), header=header, cfg=cfg,
                    dm=(c["dm_low"], c["dm_high"], c["dm_step"]), band=(first, last), ds=c["ds"],
                    t_sample=c["t_sample"])
    if c["kind"] == "stream":
        from astroflow_b200.dedisp import Stream

        hdr, first, last = _band(c)
        beam = Stream(hdr, c["dm_low"], c["dm_high"], first, last, c["dm_step"], c["ds"],
                      subband_width=c["width"], rfi=_rfi(c))
        out = beam.empty_output()
        tail = int(beam.info["tail_samples"])
        n = -(-tail // c["nsamp"])
        # the beam has been running: its tail holds earlier chunks of the same sky
        sky = _chunk((n + 1) * c["nsamp"], c["nchans"], c["nbits"], c["f_hi"], c["bandwidth"],
                     c["tsamp"], seed)
        for k in range(n):
            beam.push(sky[k * c["nsamp"]:(k + 1) * c["nsamp"]], out)
        return dict(kind="stream", beam=beam, chunk=sky[n * c["nsamp"]:].clone(), out=out)
    plan = _make_plan(c)
    return dict(kind="plan", plan=plan, x=_input(c, seed), out=plan.empty_output())


def _sums(t):
    """The sums as signed words of the same width (none reaches the sign bit)."""
    return t.view(torch.int64 if t.element_size() == 8 else torch.int32)


def run(state):
    s = state
    if s["kind"] == "plan":
        return _sums(s["plan"].run(s["x"], s["out"]))
    if s["kind"] == "stream":
        return _sums(s["beam"].push(s["chunk"], s["out"]))
    if s["kind"] == "batch":
        return [_sums(o) for o in s["batch"].run(s["xs"], s["outs"])]
    if s["kind"] == "images":
        from astroflow_b200.postprocess import device_images

        return device_images(s["sums"], s["starts"], s["counts"])
    from astroflow_b200 import _astroflow_core as core

    lo, hi, step = s["dm"]
    got = core._dedisperse_spec(s["data"], s["header"], lo, hi, s["band"][0], s["band"][1], step,
                                s["ds"], s["t_sample"], 0, "", s["cfg"])
    return list(got.dm_times)


def _plan_work(c):
    n = -(-c["nsamp"] // c["ds"])
    trials = int((c["dm_high"] - c["dm_low"]) / c["dm_step"]) + 1
    nchans = c["nchans"] - int(c["band_low"] * (c["nchans"] - 1))
    if c["algorithm"] == "brute":
        adds = trials * nchans * n
    else:
        adds = (-(-trials // 32) * nchans + trials * -(-nchans // c["width"])) * n
    out = trials * n * (8 if c["nbits"] == 32 else 4)
    return c["nsamp"] * c["nchans"] * c["nbits"] // 8, out, adds


def work(case):
    """Bytes: the chunk read once and the result written once; flops: the integer additions."""
    c = case
    if c["kind"] == "images":
        n = -(-c["cols"] // c["slice_cols"])
        return {"bytes": 4 * c["rows"] * c["cols"] + 512 * 512 * 3 * n, "flops": 2 * c["rows"] * c["cols"]}
    if c["kind"] == "batch":
        parts = [_plan_work(q) for q in _batch_cases(c)]
        return {"bytes": sum(p[0] + p[1] for p in parts), "flops": sum(p[2] for p in parts)}
    read, written, adds = _plan_work(c)
    if c["kind"] == "dropin":
        written = 512 * 512 * 3 * math.ceil(c["nsamp"] * c["tsamp"] / c["t_sample"])
    return {"bytes": read + written, "flops": adds}


def exact(case, seed):
    """Every output is a whole number or a byte: none has a 64-bit floating value."""
    return None
