"""The work that a user of skyweaver_b200 has it do, as measurable cases.

Every case goes through the package's public entry points (the stage classes
and functions of skyweaver_b200.stages, which call the C ABI), over the range
of sizes that the repository's benchmark, tests and configurations use:

  pipeline   BeamformerPipeline.process_device: one gulp through the whole
             chain (what a program that streams recordings spends its time on)
  cb         coherent_beamform_grouped: all (DM, beamset) problems of a gulp
  cdd        CoherentDedisperser.dedisperse: overlap-save FFT dedispersion
  idd        incoherent_dedisperse: trial-DM shift-and-sum over the channels
  ingest     transpose_fpact_statistics: heaps to planar rows + statistics
  ib         incoherent_beamform: incoherent beams of several beamsets
  layout     transpose_ftpa + ftpa_to_fpact: the reference's FTPA layout, which
             the C++ drop-in classes take and return

listed() names the cases, draw() gives others of the same ranges.
"""
import math

import numpy as np
import torch

from skyweaver_b200 import stages, synthetic

CHBW = 856e6 / 1024            # MeerKAT L-band channel
UHF_CHBW = 544e6 / 1024        # MeerKAT UHF channel
TONES = (9, 27, 45)            # channels with narrowband RFI, as in bench.py
EPOCH = 1.7e9
K_DM = 4.148806423e15


def listed():
    return [
        # the smallest gulp: a 16-antenna subarray, no dedispersion; launches count
        dict(name="pipeline_small", kind="pipeline", nant=16, in_nant=16, beams=64, chans=8,
             samples=4096, ts=4, dms="", stokes="I", beamsets=1, uhf=False, tones=False),
        # the benchmark's gulp: L-band subband, 4 coherent DMs, three RFI tones
        dict(name="pipeline_lband", kind="pipeline", nant=64, in_nant=64, beams=1024, chans=64,
             samples=65536, ts=16, dms="0,50,150,500", stokes="I", beamsets=1, uhf=False,
             tones=True),
        # UHF survey chain up to the beams, 57 of 64 antennas present
        dict(name="pipeline_uhf", kind="pipeline", nant=64, in_nant=57, beams=2048, chans=256,
             samples=16384, ts=8, dms="0,300", stokes="I", beamsets=1, uhf=True, tones=False),
        # 8 uneven beamsets x 4 DMs, one grouped launch
        dict(name="cb_ragged", kind="cb", nant=64, beams=1376, chans=64, samples=32768, ts=16,
             dms=4, stokes="I", beamsets=8, ib_subtract=True),
        # polarimetry at high time resolution: char4 beams, beam count off the tile
        dict(name="cb_stokes", kind="cb", nant=32, beams=200, chans=16, samples=8192, ts=4,
             dms=1, stokes="IQUV", beamsets=2, ib_subtract=False),
        # nearby pulsar: short windows (1024 points), 48 antennas, one DM
        dict(name="cdd_short", kind="cdd", nant=48, chans=32, samples=16384, dms="30",
             fft_len=0),
        # precision configuration: 65536-point windows, the largest smear
        dict(name="cdd_long", kind="cdd", nant=64, chans=8, samples=65536, dms="0,50,150,500",
             fft_len=65536),
        # coarse trials at high DM over 256 UHF channels (delays of 10^4 samples)
        dict(name="idd_uhf", kind="idd", beams=512, chans=256, samples_out=8192, trials=128,
             dm_lo=250.0, dm_hi=350.0, ts=1, base_ts=8, uhf=True),
        # fine trials at low DM over an L-band subband
        dict(name="idd_lband", kind="idd", beams=1024, chans=64, samples_out=3968, trials=32,
             dm_lo=0.0, dm_hi=10.0, ts=1, base_ts=16, uhf=False),
        # a recording's gulp into planar rows with 57 of 64 antennas, odd heap count
        dict(name="ingest", kind="ingest", nant=64, in_nant=57, chans=64, heaps=67),
        # incoherent beams of 8 beamsets (sub-array masks), short time scrunch
        dict(name="ib_beamsets", kind="ib", nant=64, chans=64, samples=32768, ts=8, beamsets=8,
             stokes="I"),
        # the reference's FTPA layout in and back to planar rows
        dict(name="layout", kind="layout", nant=64, in_nant=57, chans=16, heaps=32),
    ]


# ------------------------------------------------------------------- drawing
def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges above: kinds as often as listed, sizes over
    their logarithm, odd counts of beams, channels, heaps and trials."""
    kind = rng.choice(["pipeline", "pipeline", "pipeline", "cb", "cb", "cdd", "cdd", "idd", "idd",
                       "ingest", "ib", "layout"])
    if kind == "pipeline":
        nant = rng.choice([16, 32, 64])
        chans, beams = _log(rng, 5, 200), _log(rng, 33, 1600)
        dms = rng.choice(["", "0,%d" % rng.randint(5, 300), "%d" % rng.randint(5, 400),
                          "0,%d,%d" % (rng.randint(5, 60), rng.randint(100, 500))])
        # at most the L-band gulp's beams x channels x samples x DMs
        room = 64 * 1024 * 65536 * 4 / (chans * beams * max(1, dms.count(",") + 1))
        samples = 256 * max(8, min(256, _log(rng, 8, 256), int(room / 256)))
        return dict(kind=kind, nant=nant, in_nant=nant - rng.randint(0, nant // 4), beams=beams,
                    chans=chans, samples=samples, ts=rng.choice([4, 8, 16, 32]), dms=dms,
                    stokes=rng.choice(["I", "I", "I", "Q", "IQUV"]),
                    beamsets=rng.choice([1, 1, 3]), uhf=rng.random() < 0.3,
                    tones=rng.random() < 0.3)
    if kind == "cb":
        return dict(kind=kind, nant=rng.choice([16, 32, 64]), beams=_log(rng, 33, 1400),
                    chans=_log(rng, 3, 48), samples=64 * _log(rng, 16, 256),
                    ts=rng.choice([1, 2, 4, 8, 16, 32]), dms=rng.randint(1, 4),
                    stokes=rng.choice(["I", "I", "Q", "U", "V", "IQUV"]),
                    beamsets=rng.randint(1, 8), ib_subtract=rng.random() < 0.7)
    if kind == "cdd":
        long = rng.random() < 0.25
        dms = rng.choice(["%d", "0,%d", "0,20,%d", "10,50,90,%d"]) % rng.randint(100, 500 if long else 400)
        return dict(kind=kind, nant=rng.randint(12, 64), chans=_log(rng, 3, 12 if long else 40),
                    samples=16 * _log(rng, 256, 3000), dms=dms,
                    fft_len=rng.choice([16384, 32768, 65536]) if long else rng.choice([0, 0, 4096, 8192]))
    if kind == "idd":
        uhf = rng.random() < 0.5
        lo = rng.uniform(0.0, 250.0)
        return dict(kind=kind, beams=4 * _log(rng, 15, 160), chans=_log(rng, 24, 256 if uhf else 128),
                    samples_out=_log(rng, 200, 4000), trials=_log(rng, 5, 128), dm_lo=lo,
                    dm_hi=lo + rng.uniform(2.0, 100.0), ts=rng.choice([1, 1, 2, 4]),
                    base_ts=rng.choice([8, 16, 32]), uhf=uhf)
    nant = rng.choice([16, 32, 64])
    if kind == "ingest":
        return dict(kind=kind, nant=nant, in_nant=nant - rng.randint(0, 7), chans=_log(rng, 4, 80),
                    heaps=_log(rng, 4, 130))
    if kind == "ib":
        return dict(kind=kind, nant=nant, chans=_log(rng, 4, 64), samples=256 * _log(rng, 8, 128),
                    ts=rng.choice([4, 8, 16, 32]), beamsets=rng.randint(1, 8),
                    stokes=rng.choice(["I", "I", "Q", "IQUV"]))
    return dict(kind=kind, nant=nant, in_nant=nant - rng.randint(0, 7), chans=_log(rng, 3, 24),
                heaps=_log(rng, 3, 48))


# ----------------------------------------------------------------- geometry
def _dms(case):
    return [float(d) for d in case["dms"].split(",")] if case["dms"] else [0.0]


def _band(case):
    """(centre, bandwidth, channel bandwidth) in Hz."""
    if case.get("uhf"):  # the top channels of the 544-1088 MHz band
        bw = case["chans"] * UHF_CHBW
        return 1088e6 - bw / 2, bw, UHF_CHBW
    return 1284e6, case["chans"] * CHBW, CHBW


def _counts(case):
    """Active antennas of each beamset, falling from all of them."""
    n, a = case["beamsets"], case["nant"]
    return [max(1, a * (n - s) // n) for s in range(n)]


def _mapping(case):
    """Beam -> beamset: contiguous runs, halving like a survey's sub-arrays."""
    n, b = case["beamsets"], case["beams"]
    share = np.array([2.0 ** -s for s in range(n)])
    edge = np.round(np.cumsum(share) / share.sum() * b)
    return np.minimum(np.searchsorted(edge, np.arange(b), side="right"), n - 1).astype(np.int32)


def _cdd_geometry(case):
    """(fft_len, overlap, lag): the library's own plan for the band and DMs."""
    centre, bw, _ = _band(case)
    return stages.cdd_plan(centre, bw, case["chans"], _dms(case), fft_len=case["fft_len"])


def _idd_delays(case):
    centre, bw, chbw = _band(case)
    f = stages.channel_frequencies(centre, bw, case["chans"])
    dm = np.linspace(case["dm_lo"], case["dm_hi"], case["trials"]).astype(np.float32)
    tsamp = case["base_ts"] / chbw
    d = K_DM * (1 / f[0] ** 2 - 1 / f ** 2)[None, :] * dm[:, None].astype(np.float64) / tsamp
    return (d + 0.5).astype(np.int32)


# --------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _noise(gen, shape, sigma=8.0):
    """Rounded complex Gaussian voltages, int8, made in slabs."""
    out = torch.empty(shape, dtype=torch.int8, device="cuda")
    flat = out.view(-1)
    for lo in range(0, flat.numel(), 1 << 28):
        n = min(1 << 28, flat.numel() - lo)
        v = torch.empty(n, device="cuda").normal_(0.0, sigma, generator=gen)
        flat[lo:lo + n] = v.round_().clamp_(-127, 127).to(torch.int8)
    return out


def _taftp(gen, case, heaps):
    v = _noise(gen, (heaps, case["in_nant"], case["chans"], 256, 2, 2))
    if case.get("tones"):  # 20-sigma narrowband RFI on every antenna
        t = torch.arange(heaps * 256, device="cuda", dtype=torch.float64).reshape(heaps, 256)
        for k, c in enumerate(TONES):
            if c < case["chans"]:
                ph = 2 * math.pi * torch.remainder((0.01 + 0.037 * k) * t, 1.0)
                tone = 160.0 * torch.stack([torch.cos(ph), torch.sin(ph)], -1)
                cur = v[:, :, c].float() + tone[:, None, :, None, :].float()
                v[:, :, c] = cur.round_().clamp_(-127, 127).to(torch.int8)
    return v


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    gen, g, kind = _gen(seed), np.random.default_rng(seed), case["kind"]
    s = {"case": case}
    if kind == "pipeline":
        centre, bw, chbw = _band(case)
        masks = synthetic.beamset_masks(g, case["nant"], _counts(case))
        mapping = _mapping(case)
        delays = synthetic.delay_model(g, case["beams"], case["nant"])
        delays[..., 0] = masks[mapping]
        s["taftp"] = _taftp(gen, case, case["samples"] // 256)
        s["pipe"] = stages.BeamformerPipeline(
            nantennas=case["nant"], input_nantennas=case["in_nant"], nchans=case["chans"],
            nbeams=case["beams"], gulp_samples=case["samples"], tscrunch=case["ts"],
            centre_frequency=centre, bandwidth=bw, dms=_dms(case), beamset_weights=masks,
            beamset_mapping=mapping, stokes=case["stokes"],
            coherent_dedispersion=bool(case["dms"]))
        s["pipe"].set_delays(delays, EPOCH)
        s["masks"], s["mapping"], s["delays"] = masks, mapping, delays
        s["epoch"], s["step"] = EPOCH, case["samples"] / chbw
    elif kind == "cb":
        a, b, f, t, ts = (case[k] for k in ("nant", "beams", "chans", "samples", "ts"))
        masks = synthetic.beamset_masks(g, a, _counts(case))
        mapping = _mapping(case)
        delays = synthetic.delay_model(g, b, a)
        delays[..., 0] = masks[mapping]
        centre, bw, _ = _band(case)
        s["freqs"] = stages.channel_frequencies(centre, bw, f)
        s["delays"], s["mapping_h"] = delays, mapping
        _, s["weights"] = stages.generate_weights(_cuda(delays), _cuda(s["freqs"]), EPOCH, EPOCH,
                                                  want_fba=False)
        s["volts"] = [_noise(gen, (f, 2, a, 2, t)) for _ in range(case["dms"])]
        comp = (4,) if case["stokes"] == "IQUV" else ()
        # powers and scalings as the statistics of sigma-8 voltages give them
        n = np.repeat(np.array(_counts(case), np.float64), f)
        x, dof = (127.0 * 8.0) ** 2 * n, 4.0 * ts
        s["offset"] = _cuda((x * dof).astype(np.float32))
        s["scale"] = _cuda((x * math.sqrt(2 * dof) / 24.0).astype(np.float32))
        s["mapping"] = _cuda(mapping)
        ib = torch.empty((case["beamsets"], t // ts, f) + comp, device="cuda")
        mean = torch.tensor(np.array(_counts(case)) * 64.0 * dof, dtype=torch.float32, device="cuda")
        s["ib"] = [(ib.normal_(0.0, 0.02, generator=gen) + 1.0).mul_(
            mean.view((-1,) + (1,) * (ib.dim() - 1))).round_() for _ in range(case["dms"])]
        s["outs"] = [torch.empty((t // ts, f, b) + comp, dtype=torch.int8, device="cuda")
                     for _ in range(case["dms"])]
    elif kind == "cdd":
        centre, bw, _ = _band(case)
        n, ov, lag = _cdd_geometry(case)
        s["plan"] = (n, ov, lag)
        s["low"] = float(np.float32(centre - bw / 2))
        s["rows"] = _noise(gen, (case["chans"], 2, case["nant"], 2, ov + case["samples"]))
        s["cdd"] = stages.CoherentDedisperser(case["chans"], case["nant"], n, ov, s["low"], bw,
                                              _dms(case), lag=lag)
        s["outs"] = [torch.empty((case["chans"], 2, case["nant"], 2, case["samples"]),
                                 dtype=torch.int8, device="cuda") for _ in _dms(case)]
    elif kind == "idd":
        d = _idd_delays(case)
        s["delays"], s["maxd"] = _cuda(d), int(d.max())
        t = s["maxd"] + case["samples_out"] * case["ts"]
        s["tfb"] = _noise(gen, (t, case["chans"], case["beams"]), sigma=24.0)
        s["scale"] = float(np.float32(math.sqrt(case["chans"] * case["ts"])))
    elif kind == "ingest":
        s["taftp"] = _taftp(gen, case, case["heaps"])
    elif kind == "ib":
        s["rows"] = _noise(gen, (case["chans"], 2, case["nant"], 2, case["samples"]))
        s["masks"] = _cuda(synthetic.beamset_masks(g, case["nant"], _counts(case)))
        n = np.repeat(np.array(_counts(case), np.float64), case["chans"])
        dof = 4.0 * case["ts"]
        s["offset"] = _cuda((64.0 * n * dof).astype(np.float32))
        s["scale"] = _cuda((64.0 * np.sqrt(2 * n * dof) / 24.0).astype(np.float32))
    else:
        s["taftp"] = _taftp(gen, case, case["heaps"])
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "pipeline":
        s["pipe"].process_device(s["taftp"], s["epoch"])
        s["epoch"] += s["step"]
        beams = [s["pipe"].cb_device(d) for d in range(len(_dms(case)))]
        for b in beams:
            b.owner = s["pipe"]  # the views are the pipeline's memory: it lives as long as they
        return beams
    if kind == "cb":
        problems = [(v, o, ib if case["ib_subtract"] else None, 0, case["beams"])
                    for v, o, ib in zip(s["volts"], s["outs"], s["ib"])]
        stages.coherent_beamform_grouped(problems, s["weights"], s["scale"], s["offset"],
                                         s["mapping"], case["samples"], case["ts"],
                                         stokes=case["stokes"], ib_subtract=case["ib_subtract"])
        return s["outs"]
    if kind == "cdd":
        return s["cdd"].dedisperse(s["rows"], case["samples"], outs=s["outs"])
    if kind == "idd":
        return stages.incoherent_dedisperse(s["tfb"], s["delays"], s["maxd"], case["ts"],
                                            s["scale"])
    if kind == "ingest":
        return stages.transpose_fpact_statistics(s["taftp"], case["nant"])
    if kind == "ib":
        return stages.incoherent_beamform(s["rows"], case["samples"], case["ts"], s["scale"],
                                          s["offset"], s["masks"], stokes=case["stokes"])
    ftpa = stages.transpose_ftpa(s["taftp"], case["nant"])
    return ftpa, stages.ftpa_to_fpact(ftpa)


# ----------------------------------------------------------------------- work
def _fft_flops(streams, samples, n, ov, ninv):
    return streams * math.ceil(samples / (n - ov)) * 5.0 * n * math.log2(n) * (1 + ninv)


def work(case):
    kind = case["kind"]
    comp = 4 if case.get("stokes") == "IQUV" else 1
    if kind == "pipeline":
        a, b, f, t, ts = (case[k] for k in ("nant", "beams", "chans", "samples", "ts"))
        dms = _dms(case)
        flops = 8.0 * a * b * 2 * f * t * len(dms)
        if case["dms"]:
            centre, bw, _ = _band(case)
            n, ov, _ = stages.cdd_plan(centre, bw, f, dms)
            nz = sum(d != 0 for d in dms)
            flops += _fft_flops(f * 2 * a, t, n, ov, nz) if nz else 0.0
        return {"bytes": float(case["in_nant"] * f * t * 4 + len(dms) * (t // ts) * f * b * comp),
                "flops": flops}
    if kind == "cb":
        a, b, f, t, ts = (case[k] for k in ("nant", "beams", "chans", "samples", "ts"))
        rows = f * 4 * a * t + (t // ts) * f * b * comp
        ib = case["beamsets"] * (t // ts) * f * 4 * comp if case["ib_subtract"] else 0
        return {"bytes": float(case["dms"] * (rows + ib) + f * 4 * b * a),
                "flops": 8.0 * a * b * 2 * f * t * case["dms"]}
    if kind == "cdd":
        n, ov, _ = _cdd_geometry(case)
        f, a, t, dms = case["chans"], case["nant"], case["samples"], _dms(case)
        nz = sum(d != 0 for d in dms)
        return {"bytes": float(f * 4 * a * (ov + t * (1 + len(dms)))),
                "flops": _fft_flops(f * 2 * a, t, n, ov, nz)}
    if kind == "idd":
        f, b, o, d = case["chans"], case["beams"], case["samples_out"], case["trials"]
        t = int(_idd_delays(case).max()) + o * case["ts"]
        return {"bytes": float(t * f * b + o * d * b), "flops": float(o * case["ts"]) * d * f * b}
    if kind == "ib":
        f, a, t, ts, n = (case[k] for k in ("chans", "nant", "samples", "ts", "beamsets"))
        return {"bytes": float(f * 4 * a * t + 5 * n * (t // ts) * f * comp),
                "flops": float(f * a * t) * (8 + 2 * n) * comp}
    v = float(case["heaps"] * 256 * case["chans"] * 4)
    if kind == "ingest":
        return {"bytes": v * (case["in_nant"] + case["nant"]), "flops": 8 * v * case["in_nant"]}
    return {"bytes": v * (case["in_nant"] + 2 * case["nant"]), "flops": 0.0}


def tolerance(case):
    kind = case["kind"]
    # int8 outputs: shares of values that fall to the other side of a rounding
    # boundary, four times what the 64-bit results were seen to differ by
    # (pipeline 2.8e-4, one dedispersed voltage in 10^6 reaching 1024 beams;
    # cdd 1.8e-6, cb 8.4e-6, ib 3.9e-4)
    if kind == "pipeline":
        return {"rel": 1e-5, "differ": 1.2e-3}
    if kind == "cdd":
        return {"rel": 1e-5, "differ": 8e-6}
    if kind == "cb":
        return {"rel": 1e-5, "differ": 3e-5}
    if kind == "ingest":
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "ib":
        return {"rel": 1e-6, "max": 1e-5, "differ": 1.6e-3}
    return "exact"


# ---------------------------------------------------------------- 64 bits
def _planes(rows):
    """int8 [..., re|im, t] -> complex128 [..., t]."""
    return torch.complex(rows[..., 0, :].double(), rows[..., 1, :].double())


def _to_rows(z):
    """complex [..., t] of whole numbers -> int8 [..., re|im, t] (wrapping)."""
    return torch.stack([z.real, z.imag], -2).round().to(torch.int32).to(torch.int8)


def _fpact64(taftp, nant):
    """TAFTP -> FPACT int8 [F][2][nant][2][T]."""
    h, a, f = taftp.shape[:3]
    out = torch.zeros((f, 2, nant, 2, h * 256), dtype=torch.int8, device=taftp.device)
    out[:, :, :a] = taftp.permute(2, 4, 1, 5, 0, 3).reshape(f, 2, a, 2, h * 256)
    return out


def _chirp64(chans, c, n, low, bw, dm):
    cbw = bw / chans
    nu0 = low + c * cbw - 0.5 * cbw
    nu = torch.arange(n, dtype=torch.float64, device="cuda") * (cbw / n)
    ph = -2.0 * math.pi * K_DM * float(np.float32(dm)) * nu * nu / ((nu0 + nu) * nu0 * nu0)
    return torch.complex(torch.cos(ph), torch.sin(ph))


def _cdd64(rows, samples, n, ov, lag, chirp):
    """Overlap-save of one channel: int8 [P][A][2][ov + samples] -> same, samples."""
    z = _planes(rows)
    step, out = n - ov, torch.empty(z.shape[:-1] + (samples,), dtype=z.dtype, device=z.device)
    for start in range(0, samples, step):
        w = z[..., start:start + n]
        if w.shape[-1] < n:
            w = torch.nn.functional.pad(w, (0, n - w.shape[-1]))
        y = torch.fft.ifft(torch.fft.fft(w) * chirp)[..., ov - lag:ov - lag + step]
        out[..., start:start + step] = y[..., :samples - start]
    return _to_rows(out)


def _stokes64(p0, p1, stokes):
    """[...] complex voltages of both pols -> float64 [..., component]."""
    i0, i1 = p0.abs() ** 2, p1.abs() ** 2
    x = 2 * p0 * p1.conj()
    every = {"I": i0 + i1, "Q": i0 - i1, "U": x.real, "V": x.imag}
    return torch.stack([every[c] for c in stokes], -1)


def _scrunch(x, ts):
    """[T][...] -> [T / ts][...]"""
    return x.view((x.shape[0] // ts, ts) + x.shape[1:]).sum(1)


def _int8(x):
    return x.round().clamp(-128, 127).to(torch.int8)


def _ib64(rows, ts, masks, stokes):
    """One channel's incoherent power float64 [S][T/ts][component]."""
    z = _planes(rows)
    st = _stokes64(z[0].T, z[1].T, stokes)                  # [T][A][C]
    return torch.stack([_scrunch((st * m.double()[None, :, None]).sum(1), ts) for m in masks])


def _weights64(delays, freq, dt):
    d = _cuda(delays).double()
    ph = 2 * math.pi * (dt * d[..., 2] + d[..., 1]) * freq
    re, im = torch.cos(ph) * 127.0 * d[..., 0], -torch.sin(ph) * 127.0 * d[..., 0]
    return torch.complex(re.round().clamp(-128, 127), im.round().clamp(-128, 127))


def _cb64(rows, w, ts, stokes, mapping, scale, offset, ib):
    """One channel's coherent beams int8 [T/ts][B][component]; ib float64
    [S][T/ts][component] or None; scale, offset float64 [S]."""
    z, out = _planes(rows), []
    for lo in range(0, z.shape[-1], 4096):
        v = z[..., lo:lo + 4096]
        p = [w @ v[k] for k in (0, 1)]                                   # [B][t]
        out.append(_scrunch(_stokes64(p[0].T, p[1].T, stokes), ts))      # [t/ts][B][C]
    power, sc = torch.cat(out), scale[mapping][None, :, None]
    if ib is not None:
        power = power - 16129.0 * ib[mapping].transpose(0, 1)
    elif stokes[0] == "I":
        power[..., 0] -= offset[mapping][None, :]
    return _int8(power / sc)


def _pipeline64(case, s):
    centre, bw, _ = _band(case)
    f, a, t, ts, dms = case["chans"], case["nant"], case["samples"], case["ts"], _dms(case)
    stokes = case["stokes"]
    freqs = stages.channel_frequencies(centre, bw, f)
    masks, mapping = _cuda(s["masks"]).double(), _cuda(s["mapping"]).long()
    n, ov, lag = stages.cdd_plan(centre, bw, f, dms) if case["dms"] else (0, 0, 0)
    low = float(np.float32(centre - bw / 2))
    outs = [torch.empty((t // ts, f, case["beams"], len(stokes)), dtype=torch.int8, device="cuda")
            for _ in dms]
    for c in range(f):
        rows = _fpact64(s["taftp"][:, :, c:c + 1], a)[0]
        x = rows.permute(0, 1, 3, 2).reshape(2, a, -1).double()
        std = x.std(-1)                                                  # [P][A]
        count = 2.0 * masks.sum(1)
        avg, eff = (masks @ std.sum(0)) / count, count / 2.0
        dof = 4.0 * ts
        cb = (127.0 * avg) ** 2 * eff
        ext = torch.nn.functional.pad(rows, (ov, 0))
        w = _weights64(s["delays"], freqs[c], 0.0)
        for d, dm in enumerate(dms):
            if dm == 0.0:
                v = ext[..., ov - lag:ov - lag + t]
            else:
                v = _cdd64(ext, t, n, ov, lag, _chirp64(f, c, n, low, bw, dm))
            ib = _ib64(v, ts, masks, stokes)
            outs[d][:, c] = _cb64(v, w, ts, stokes, mapping, cb * math.sqrt(2 * dof) / 24.0,
                                  cb * dof, ib)
    return [o if len(stokes) > 1 else o[..., 0] for o in outs]


def exact(case, seed):
    """run() on the same inputs in 64 bits with torch alone."""
    kind, s = case["kind"], prepare(case, seed)
    if kind == "pipeline":
        return _pipeline64(case, s)
    if kind == "cb":
        f, a, b = case["chans"], case["nant"], case["beams"]
        stokes, mapping = case["stokes"], s["mapping"].long()
        scale, offset = (s[k].double().view(-1, f) for k in ("scale", "offset"))
        outs = []
        for v, ib in zip(s["volts"], s["ib"]):
            ib = ib.double() if len(stokes) > 1 else ib.double()[..., None]
            o = torch.stack([_cb64(v[c], _weights64(s["delays"], s["freqs"][c], 0.0), case["ts"],
                                   stokes, mapping, scale[:, c], offset[:, c],
                                   ib[:, :, c] if case["ib_subtract"] else None)
                             for c in range(f)], 1)
            outs.append(o if len(stokes) > 1 else o[..., 0])
        return outs
    if kind == "cdd":
        _, bw, _ = _band(case)
        n, ov, lag = s["plan"]
        return [torch.stack([_cdd64(s["rows"][c], case["samples"], n, ov, lag,
                                    _chirp64(case["chans"], c, n, s["low"], bw, dm))
                             for c in range(case["chans"])]) for dm in _dms(case)]
    if kind == "idd":
        o, ts, d = case["samples_out"], case["ts"], s["delays"].cpu().numpy()
        out = torch.empty((o, case["trials"], case["beams"]), dtype=torch.int8, device="cuda")
        for k in range(case["trials"]):
            acc = torch.zeros((o * ts, case["beams"]), dtype=torch.int32, device="cuda")
            for c in range(case["chans"]):
                lo = s["maxd"] - int(d[k, c])
                acc += s["tfb"][lo:lo + o * ts, c]
            v = _scrunch(acc, ts).double() / s["scale"]
            out[:, k] = v.trunc().clamp(-128, 127).to(torch.int8)
        return out
    if kind == "ingest":
        rows = _fpact64(s["taftp"], case["nant"])
        x = rows.reshape(rows.shape[:3] + (-1,)).double()
        n, m = x.shape[-1], x.mean(-1, keepdim=True)
        d = x - m
        m2, m3, m4 = ((d ** k).sum(-1) for k in (2, 3, 4))
        st = torch.stack([m[..., 0], (m2 / (n - 1)).sqrt(), math.sqrt(n) * m3 / m2 ** 1.5,
                          n * m4 / (m2 * m2) - 3.0], -1)
        return rows, st
    if kind == "ib":
        f, stokes = case["chans"], case["stokes"]
        scale, offset = (s[k].double().view(-1, 1, f, 1) for k in ("scale", "offset"))
        raw = torch.stack([_ib64(s["rows"][c], case["ts"], s["masks"], stokes) for c in range(f)], 2)
        lessened = raw.clone()
        if stokes[0] == "I":
            lessened[..., :1] -= offset
        out = _int8(lessened / scale)
        return (raw, out) if len(stokes) > 1 else (raw[..., 0], out[..., 0])
    rows = _fpact64(s["taftp"], case["nant"])
    ftpa = rows.permute(0, 4, 1, 2, 3).contiguous()
    return ftpa, rows
