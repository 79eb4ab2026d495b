"""Kernel variants and dispatch rules at the sizes where they can go wrong:
tile edges, remainders, the smallest and largest of their ranges."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(cuda, a):
    return cuda.from_numpy(np.ascontiguousarray(a)).cuda()


def _np(t):
    return t.cpu().numpy()


@pytest.mark.parametrize("nant,T,stride,off", [
    (64, 128, 128, 0), (64, 131, 144, 13), (1, 1, 1, 0), (13, 127, 128, 0), (65, 130, 132, 0),
    (200, 257, 272, 12), (32, 4, 7, 3)])
def test_layout_converters_ragged(cuda, nant, T, stride, off):
    """FTPA <-> FPACT for antenna counts and sample counts off the 64 x 128
    tile, rows off the 4-byte grid: the bytes outside [off, off + T) stay."""
    from skyweaver_b200 import stages
    g = np.random.default_rng(nant * 1000 + T)
    F = 3
    ftpa = g.integers(-128, 128, size=(F, T, 2, nant, 2), dtype=np.int8)
    fp = stages.ftpa_to_fpact(_dev(cuda, ftpa), row_stride=stride, offset=off)
    ref = np.zeros((F, 2, nant, 2, stride), np.int8)
    ref[..., off:off + T] = ftpa.transpose(0, 2, 3, 4, 1)
    assert np.array_equal(_np(fp), ref)
    assert np.array_equal(_np(stages.fpact_to_ftpa(fp, T, offset=off)), ftpa)


@pytest.mark.parametrize("F,nant,T,stride,off", [
    (1, 1, 40000, 40004, 4), (5, 2, 5003, 5003, 0), (2, 6, 4096, 4112, 13),  # a thread per antenna
    (40, 7, 5, 8, 0), (80, 7, 250, 256, 3),          # past that: tiles
    (23, 64, 128, 128, 0), (24, 64, 128, 128, 0),    # on either side of the tile counts that
    (147, 64, 128, 131, 1), (148, 64, 128, 131, 1),  # part them, rows on and off the 4-byte grid
    (160, 64, 131, 144, 13), (75, 65, 130, 132, 0), (40, 250, 129, 131, 1)])
def test_layout_converters_forms(cuda, F, nant, T, stride, off):
    """Both forms of the FTPA <-> FPACT converters at the lines between them,
    whole and ragged tiles, rows on and off the 4-byte grid: equal to the
    permutation, and the bytes outside [off, off + T) stay."""
    from skyweaver_b200 import stages
    torch = cuda
    gen = torch.Generator(device="cuda").manual_seed(F + nant)
    ftpa = torch.randint(-128, 128, (F, T, 2, nant, 2), dtype=torch.int8, device="cuda", generator=gen)
    fp = stages.ftpa_to_fpact(ftpa, row_stride=stride, offset=off)
    ref = torch.zeros((F, 2, nant, 2, stride), dtype=torch.int8, device="cuda")
    ref[..., off:off + T] = ftpa.permute(0, 2, 3, 4, 1)
    assert torch.equal(fp, ref)
    assert torch.equal(stages.fpact_to_ftpa(fp, T, offset=off), ftpa)


@pytest.mark.parametrize("ts,stokes", [(1, "I"), (4, "Q"), (16, "I"), (2, "IQUV"), (32, "V")])
@pytest.mark.parametrize("ib_sub", [True, False])
def test_coherent_beam_quantiser(cuda, oracle, ts, stokes, ib_sub):
    """The divisionless quantiser against the reference's division where it
    could err: small whole powers over scales that put many quotients on or
    next to half-integers, quotients far outside the clamp, negative scales
    and scales whose reciprocal is subnormal or overflows (bit-exact)."""
    from skyweaver_b200 import stages
    g = np.random.default_rng(5 + ts)
    A, B, T = 16, 40, 512
    scl = np.array([2.0, -2.0, 6.0, 7.0, 48.0, 0.37, 1e-35, 1e-39, 3e33, 1e-30, 254.0, 1000.0],
                   np.float32)
    F = len(scl)
    ftpa = g.integers(-2, 3, size=(F, T, 2, A, 2), dtype=np.int8)
    w = g.integers(-1, 2, size=(F, B, A, 2), dtype=np.int8)
    bw = np.ones((1, A), np.float32)
    off = np.full(F, 100.0, np.float32)
    mapping = np.zeros(B, np.int32)
    ref = oracle.coherent_beam(ftpa, w, ts, scl, off, bw, mapping, stokes, ib_sub)
    fp = stages.ftpa_to_fpact(_dev(cuda, ftpa))
    raw = None
    if ib_sub:
        one = _dev(cuda, np.ones(F, np.float32))
        raw, _ = stages.incoherent_beamform(fp, T, ts, one, one, _dev(cuda, bw), stokes=stokes)
    out = stages.coherent_beamform(fp, stages.pack_weights(_dev(cuda, w)), _dev(cuda, scl),
                                   _dev(cuda, off), _dev(cuda, mapping), raw, T, ts,
                                   stokes=stokes, ib_subtract=ib_sub)
    assert np.array_equal(_np(out), ref)


@pytest.mark.parametrize("ts,stokes", [(1, "I"), (2, "Q"), (4, "I"), (8, "U"), (8, "IQUV"),
                                       (16, "IQUV"), (16, "I"), (32, "I")])
def test_coherent_beam_lanes_part(cuda, oracle, ts, stokes):
    """Beamsets that alternate from lane to lane, some of whose outputs are all
    divided, some never, and beams missing from the last warps: every column
    group after them is loaded by the whole warp (bit-exact)."""
    from skyweaver_b200 import stages
    g = np.random.default_rng(ts)
    A, B, T, F, S = 16, 45, 1024, 3, 4
    ftpa = g.integers(-2, 3, size=(F, T, 2, A, 2), dtype=np.int8)
    w = g.integers(-1, 2, size=(F, B, A, 2), dtype=np.int8)
    bw = np.ones((S, A), np.float32)
    scl = np.repeat(np.array([2.0, 1e-35, 48.0, 7.0], np.float32), F)
    off = np.full(S * F, 100.0, np.float32)
    mapping = (np.arange(B) % S).astype(np.int32)
    ref = oracle.coherent_beam(ftpa, w, ts, scl, off, bw, mapping, stokes, False)
    out = stages.coherent_beamform(stages.ftpa_to_fpact(_dev(cuda, ftpa)),
                                   stages.pack_weights(_dev(cuda, w)), _dev(cuda, scl),
                                   _dev(cuda, off), _dev(cuda, mapping), None, T, ts,
                                   stokes=stokes, ib_subtract=False)
    assert np.array_equal(_np(out), ref)


@pytest.mark.parametrize("B,F,T", [(1, 1, 64), (129, 2, 64), (64, 8, 4096), (300, 5, 1216),
                                   (128, 149, 128), (257, 37, 8256)])
def test_coherent_beam_default_work_items(cuda, B, F, T):
    """The default work-item size (by the launch's size) gives the bytes that
    one tile per item and the longest items give."""
    from skyweaver_b200 import stages
    g = np.random.default_rng(B + F)
    A, ts = 32, 4
    fp = _dev(cuda, g.integers(-60, 61, size=(F, 2, A, 2, T), dtype=np.int8))
    w = _dev(cuda, g.integers(-127, 128, size=(F, 2, B, A, 2), dtype=np.int8))
    scl = _dev(cuda, np.full(F, 3e7, np.float32))
    off = _dev(cuda, np.full(F, 1e9, np.float32))
    mapping = _dev(cuda, np.zeros(B, np.int32))
    out = [_np(stages.coherent_beamform(fp, w, scl, off, mapping, None, T, ts, ib_subtract=False,
                                        tiles_per_item=n)) for n in (0, 1, 1024)]
    assert np.array_equal(out[0], out[1]) and np.array_equal(out[0], out[2])


@pytest.mark.parametrize("n,F,P,A,T,ov,lag,dms,pad", [
    (8192, 1, 2, 1, 7000, 1600, 128, [500.0], 0),          # one window
    (8192, 2, 2, 37, 6593, 1600, 128, [50.0, 500.0], 7),   # odd samples and stride: byte stores
    (8192, 1, 1, 3, 20000, 1333, 401, [0.0, 333.0], 16),   # odd overlap and lag, odd window count
    (8192, 3, 2, 50, 16, 48, 16, [3.0, 0.0, 2.0], 0),      # a few samples; more windows than SMs
    (8192, 2, 2, 4, 40000, 8000, 4000, [150.0], 2),        # 192 useful samples per window
    (4096, 2, 2, 5, 9001, 1334, 400, [0.0, 100.0, 300.0], 3),
    (4096, 3, 2, 64, 3000, 96, 16, [20.0], 8),
    (2048, 3, 2, 33, 5000, 501, 77, [10.0, 0.0], 1),
    (2048, 1, 1, 1, 64, 32, 16, [1.0], 0),
    (1024, 2, 2, 21, 10000, 240, 128, [5.0, 30.0], 4),
    (1024, 1, 2, 7, 2001, 111, 30, [0.0, 7.0], 3),
    (512, 2, 2, 9, 3000, 97, 20, [3.0], 1),
    (16384, 1, 2, 3, 20001, 1601, 129, [0.0, 300.0], 3),   # split transforms
    (32768, 2, 1, 2, 5000, 3000, 128, [0.0, 400.0], 0),
    (65536, 1, 2, 2, 70000, 1600, 128, [500.0, 0.0, 50.0], 6),
])
def test_coherent_dedispersion_windows(cuda, n, F, P, A, T, ov, lag, dms, pad):
    """Windows of every length at odd trims, strides and window counts against
    torch's FP64 transform: bytes differ only where the FP64 value lies within
    the transform's single-precision error of a half-integer, and the float
    outputs by no more than that.  The error bound is log2 n butterfly stages
    of 2^-24 each way on values of rms 12 sqrt(2), times 8 for the largest of
    10^6."""
    from skyweaver_b200 import stages
    torch = cuda
    g = np.random.default_rng(T + ov)
    chbw = 856e6 / 1024
    bw, low = F * chbw, 1257e6
    tol = 8 * 2 * np.log2(n) * 2.0 ** -24 * 17.0
    ext = np.clip(np.rint(g.normal(0, 12, size=(F, P, A, 2, ov + T + pad))), -127, 127)
    ext = _dev(cuda, ext.astype(np.int8))
    cdd = stages.CoherentDedisperser(F, A, n, ov, low, bw, dms, lag=lag)
    outs = [torch.full((F, P, A, 2, T + pad), 99, dtype=torch.int8, device="cuda") for _ in dms]
    plain = [o.clone() for o in outs]
    _, dbg = cdd.dedisperse(ext, T, outs=outs, debug=True)
    # long windows: one at a time through the smallest workspace
    cdd.dedisperse(ext, T, outs=plain, workspace_limit=1)
    z = torch.complex(ext[..., 0, :ov + T].double(), ext[..., 1, :ov + T].double())
    step = n - ov
    for d, dm in enumerate(dms):
        k = torch.arange(n, dtype=torch.float64, device="cuda") * (chbw / n)
        nu0 = (low + (torch.arange(F, dtype=torch.float64, device="cuda") - 0.5) * chbw)[:, None]
        ph = -2 * np.pi * 4.148806423e15 * float(np.float32(dm)) * k * k / ((nu0 + k) * nu0 * nu0)
        chirp = torch.polar(torch.ones_like(ph), ph)[:, None, None]
        ref = torch.empty((F, P, A, T), dtype=torch.complex128, device="cuda")
        for s in range(0, T, step):
            win = torch.nn.functional.pad(z[..., s:s + n], (0, max(0, s + n - z.shape[-1])))
            y = torch.fft.ifft(torch.fft.fft(win) * chirp)[..., ov - lag:ov - lag + step]
            ref[..., s:s + step] = y[..., :T - s]
        r = torch.stack([ref.real, ref.imag], -2)
        for o in (outs[d], plain[d]):
            assert bool((o[..., T:] == 99).all())
            err = (o[..., :T].double() - r).abs()
            assert float(err.max()) <= 0.5 + tol, (dm, float(err.max()))
        f = torch.view_as_complex(dbg[d]).to(torch.complex128)
        assert float((f - ref).abs().max()) <= tol


@pytest.mark.parametrize("n", [1024, 2048, 4096, 8192, 16384])
@pytest.mark.parametrize("T,pad,lag", [(37, 0, 16), (5001, 7, 19), (2047, 2, 0)])
def test_coherent_dedispersion_uneven_lanes(cuda, n, T, pad, lag):
    """Copies of zero DMs, staging and trimmed stores that end inside a warp,
    before its barriers and tensor memory accesses: the bytes of the same
    samples in rows where all lanes end together, launch after launch."""
    from skyweaver_b200 import stages
    torch = cuda
    ov, chbw, F, A = 208, 856e6 / 1024, 2, 37
    dms = [0.0, 4.0, 0.0, 9.0]
    g = np.random.default_rng(n + T)
    T16, ov16 = -(-T // 16) * 16, ov
    rows = np.zeros((F, 2, A, 2, ov16 + T16), np.int8)
    rows[..., :ov + T] = np.rint(g.normal(0, 12, size=(F, 2, A, 2, ov + T)))
    even = _dev(cuda, rows)
    uneven = _dev(cuda, np.ascontiguousarray(rows[..., :ov + T + pad]) if ov + T + pad <= rows.shape[-1]
                  else np.pad(rows[..., :ov + T], [(0, 0)] * 4 + [(0, pad)]))
    cdd = stages.CoherentDedisperser(F, A, n, ov, 1257e6, F * chbw, dms, lag=lag)
    ref = cdd.dedisperse(even, T16)
    for _ in range(3):
        outs = [torch.full((F, 2, A, 2, T + pad), 99, dtype=torch.int8, device="cuda") for _ in dms]
        cdd.dedisperse(uneven, T, outs=outs)
        for o, r in zip(outs, ref):
            assert torch.equal(o[..., :T], r[..., :T]) and bool((o[..., T:] == 99).all())


@pytest.mark.parametrize("n", [1024, 2048, 4096, 8192])
@pytest.mark.parametrize("T,ndms", [(200, 8), (3000, 3), (9000, 33)])
def test_coherent_dedispersion_splits_dms(cuda, n, T, ndms):
    """A launch of few windows gives a window's DMs to several groups of
    threads: the same bytes as in a launch that is too large for that, DMs of 0
    in any place (from the 33rd on they are transformed)."""
    from skyweaver_b200 import stages
    torch = cuda
    ov, lag, chbw = 224, 48, 856e6 / 1024
    dms = [0.0 if d % 5 == 1 else 0.05 * d for d in range(ndms)]
    g = np.random.default_rng(n + T)
    one = _dev(cuda, np.rint(g.normal(0, 12, size=(1, 1, 2, 2, ov + T))).astype(np.int8))
    many = one.repeat(1, 1, 400, 1, 1)
    cdd = stages.CoherentDedisperser(1, 2, n, ov, 1257e6, chbw, dms, lag=lag)
    small, large = cdd.dedisperse(one, T), cdd.dedisperse(many, T)
    for d in range(ndms):
        assert torch.equal(large[d], small[d].repeat(1, 1, 400, 1, 1)), d
        if dms[d] == 0.0 and d < 32:
            assert torch.equal(small[d], one[..., ov - lag:ov - lag + T])


@pytest.mark.parametrize("n", [512, 1024, 4096, 8192, 16384])
def test_coherent_dedispersion_without_a_number(cuda, n):
    """A chirp with a bin that is no number (a DM that is none; in a band from
    0 Hz the first channel's bin at 0 Hz, where the phase is a division by 0)
    reaches every sample of that channel: no numbers in the float output, zeros
    in the bytes, and nothing in the other channels and DMs."""
    from skyweaver_b200 import stages
    torch = cuda
    F, A, T, ov = 2, 3, 900, 64
    g = np.random.default_rng(n)
    ext = _dev(cuda, np.rint(g.normal(0, 20, size=(F, 2, A, 2, ov + T))).astype(np.int8))
    nan, inf = float("nan"), float("inf")
    for low, dms, none in ((0.0, [1e-9, 2e-9], [[0], [0]]), (1257e6, [30.0, nan, inf], [[], [0, 1], [0, 1]])):
        cdd = stages.CoherentDedisperser(F, A, n, ov, low, F * 856e6 / 1024, dms, lag=16)
        outs, dbg = cdd.dedisperse(ext, T, debug=True)
        plain = cdd.dedisperse(ext, T)
        for d, channels in enumerate(none):
            for f in range(F):
                assert bool(torch.isnan(dbg[d, f]).all() if f in channels
                            else torch.isfinite(dbg[d, f]).all())
                for o in (outs, plain):
                    assert bool((o[d][f] == 0).all()) == (f in channels)


@pytest.mark.parametrize("A,T,ts,S,stokes,sigma", [
    (1, 16, 16, 1, "I", 8), (3, 48, 4, 1, "Q", 8), (65, 1040, 8, 9, "I", 8), (200, 544, 32, 2, "V", 8),
    (64, 528, 16, 8, "IQUV", 8), (7, 2064, 4, 3, "IQUV", 60), (64, 512, 8, 2, "I", 90),
    (70, 64, 32, 1, "U", 90), (16, 32, 4, 5, "I", 127), (100, 2064, 4, 2, "IQUV", 60),
    (65, 1040, 8, 1, "Q", 60), (256, 80, 16, 1, "I", 40), (128, 32, 32, 2, "V", 90)])
@pytest.mark.parametrize("weights", ["masks", "large", "fractional"])
def test_incoherent_beam_runs(cuda, oracle, A, T, ts, S, stokes, sigma, weights):
    """The 16-sample-run form against the oracle and against the general form
    (rows off the 16-byte grid) at ragged run counts, antenna counts off the
    four warps and the chain's table, more beamsets than a pass takes, signals
    on both sides of the exactness bound and weights that are not whole."""
    from skyweaver_b200 import stages
    g = np.random.default_rng(A + T + ts)
    F = 3
    ftpa = np.clip(np.rint(g.normal(0, sigma, size=(F, T, 2, A, 2))), -128, 127).astype(np.int8)
    ftpa[1] = np.clip(ftpa[1].astype(int) * 4, -128, 127)
    bw = {"masks": g.integers(0, 2, size=(S, A)), "large": g.integers(-900, 901, size=(S, A)),
          "fractional": g.uniform(0, 1, size=(S, A))}[weights].astype(np.float32)
    scale = g.uniform(50, 5e4, size=S * F).astype(np.float32)
    offset = g.uniform(0, 1e5, size=S * F).astype(np.float32)
    args = [_dev(cuda, x) for x in (scale, offset, bw)]
    raw_ref, out_ref = oracle.incoherent_beam(ftpa, ts, scale, offset, bw, S, stokes)
    for stride, off in ((T, 0), (T + 16, 16), (T + 12, 4)):
        fp = stages.ftpa_to_fpact(_dev(cuda, ftpa), row_stride=stride, offset=off)
        raw, out = stages.incoherent_beamform(fp, T, ts, *args, offset_samples=off, stokes=stokes)
        assert np.array_equal(_np(raw), raw_ref), (stride, off)
        assert np.array_equal(_np(out), out_ref), (stride, off)


@pytest.mark.parametrize("H,A_in,A,F", [(1, 1, 4, 1), (1, 13, 16, 3), (9, 62, 64, 2), (67, 57, 64, 5),
                                        (16, 255, 256, 1), (8, 5, 5, 160)])
def test_transpose_statistics_splits(cuda, H, A_in, A, F):
    """The fused pass at every way its launch splits heaps and antenna groups
    equals the separate stages."""
    from skyweaver_b200 import stages
    g = np.random.default_rng(H * A + F)
    taftp = _dev(cuda, g.integers(-128, 128, size=(H, A_in, F, 256, 2, 2), dtype=np.int8))
    fp, st = stages.transpose_fpact_statistics(taftp, A)
    ref = stages.transpose_fpact(taftp, A)
    assert bool((fp == ref).all())
    assert np.array_equal(_np(st), _np(stages.statistics(ref, H * 256)), equal_nan=True)


@pytest.mark.parametrize("H,A_in,A,F", [(2048, 1, 8, 1), (3, 24, 24, 683), (2, 24, 24, 1023),
                                        (3, 25, 32, 683), (2, 255, 256, 3)])
def test_transpose_ftpa_parts(cuda, H, A_in, A, F):
    """Whole and half heaps per CTA on either side of the antenna and CTA
    counts that part them, antennas absent and the most there can be."""
    from skyweaver_b200 import stages
    torch = cuda
    gen = torch.Generator(device="cuda").manual_seed(H + A)
    taftp = torch.randint(-128, 128, (H, A_in, F, 256, 2, 2), dtype=torch.int8, device="cuda",
                          generator=gen)
    ref = torch.zeros((F, H, 256, 2, A, 2), dtype=torch.int8, device="cuda")
    ref[:, :, :, :, :A_in] = taftp.permute(2, 0, 3, 4, 1, 5)
    assert torch.equal(stages.transpose_ftpa(taftp, A), ref.view(F, H * 256, 2, A, 2))


@pytest.mark.parametrize("scale,rate,age", [(1e-6, 0.0, 0.0), (3e-5, 1e-9, 3600.0), (20.0, 0.0, 0.0)])
def test_weights_single_precision_path(cuda, scale, rate, age):
    """Weights on the single-precision path, near half-integers (phases whose
    cosine times 127 a is one) and past its range of turns equal the FP64
    formula (WeightsManager.cu:16-87, clamped to int8), for antenna weights
    other than 0 and 1 too.  FP64 values within 1e-9 of a half-integer, where
    the host's and the device's last bits decide, are left out."""
    from skyweaver_b200 import stages
    g = np.random.default_rng(11)
    B, A = 40, 64
    freqs = np.array([1284e6, 1e9, 544e6 + 0.25])
    d = np.zeros((B, A, 3), np.float32)
    d[..., 0] = g.choice([0.0, 1.0, 0.5, -1.0, 1.7, 30.0, 6000.0], size=(B, A))
    d[..., 1] = g.uniform(-scale, scale, size=(B, A))
    d[..., 2] = g.uniform(-rate, rate, size=(B, A))
    # 127 cos(2 pi phase) on half-integers at the second frequency
    half = np.arccos((g.integers(-127, 127, size=(10, A)) + 0.5) / 127) / (2 * np.pi)
    d[:10, :, 0], d[:10, :, 1] = 1.0, half / freqs[1]
    fba, gemm = stages.generate_weights(_dev(cuda, d), _dev(cuda, freqs), 1.7e9 + age, 1.7e9)
    D = d.astype(np.float64)
    phase = (age * D[..., 2] + D[..., 1])[None] * freqs[:, None, None]
    w = np.stack([np.cos(6.283185307179586 * phase) * 127.0 * D[..., 0],
                  -np.sin(6.283185307179586 * phase) * 127.0 * D[..., 0]], -1)
    clear = np.abs(np.abs(w - np.rint(w)) - 0.5) > 1e-9
    assert clear.mean() > 0.999
    ref = np.clip(np.rint(w), -128, 127).astype(np.int8)
    assert np.array_equal(_np(fba)[clear], ref[clear])
    assert np.array_equal(_np(stages.pack_weights(fba)), _np(gemm))


@pytest.mark.parametrize("B", [16, 24, 20, 4, 516, 1040])
@pytest.mark.parametrize("scale", [1.0, 8.0, 3.0, 6.0, 11.313708, 0.25, 1e-35, 1e33, -4.0, 2.9999998])
def test_incoherent_dedispersion_quantiser(cuda, oracle, B, scale):
    """Every load width of the dedisperser, partial last lanes, and the
    divisionless truncation against the oracle's division: scales with many
    whole quotients, quotients next to whole numbers, saturated ones, negative
    scales and scales whose reciprocal is subnormal or overflows."""
    from skyweaver_b200 import stages
    g = np.random.default_rng(B)
    F, D, ts, nout, maxd = 11, 3, 2, 37, 9
    delays = g.integers(0, maxd + 1, size=(D, F)).astype(np.int32)
    delays[0, 0] = maxd
    T = maxd + nout * ts
    tfb = np.rint(g.normal(0, 12, size=(T, F, B))).clip(-128, 127).astype(np.int8)
    tfb[: T // 3] = 127
    ref = oracle.idd(tfb, delays, maxd, ts, np.float32(scale))
    got = stages.incoherent_dedisperse(_dev(cuda, tfb), _dev(cuda, delays), maxd, ts, scale)
    assert np.array_equal(_np(got), ref)


@pytest.mark.parametrize("scale", [1.0, 3.0, 0.37, 2.9999998, -1.0, 7.0])
def test_incoherent_dedispersion_saturated(cuda, oracle, scale):
    """Sums on, next to and far beyond the quantiser's limits (quotients of
    127, 128, -128, -129 and their neighbours by one unit of the sum, and all
    128 x 11 of the largest sums) against the oracle's division."""
    from skyweaver_b200 import stages
    F, D, B, maxd = 11, 2, 64, 3
    want = sorted({s for q in (126, 127, 128, 129, 200, 1397) for e in (-1, 0, 1)
                   for s in (int(q * abs(scale)) + e, -int(q * abs(scale)) + e)
                   if abs(s) <= 127 * F})
    nout = -(-len(want) // B)
    sums = np.resize(np.array(want), nout * B).reshape(nout, B)
    tfb = np.zeros((maxd + nout, F, B), np.int64)
    left = np.zeros((maxd + nout, B), np.int64)
    left[maxd:] = sums
    for f in range(F):  # spread each sum over the channels
        tfb[:, f] = np.clip(left, -127, 127)
        left -= tfb[:, f]
    assert not left.any()
    tfb = tfb.astype(np.int8)
    delays = np.zeros((D, F), np.int32)
    delays[1, ::2] = maxd
    ref = oracle.idd(tfb, delays, maxd, 1, np.float32(scale))
    got = stages.incoherent_dedisperse(_dev(cuda, tfb), _dev(cuda, delays), maxd, 1, scale)
    assert np.array_equal(_np(got), ref)


def _idd_rows(torch, tfb, delays, max_delay, ts, scale, lo, hi):
    """Outputs lo .. hi - 1 in plain torch: sums in int32, one float division,
    truncation and clamp."""
    out = []
    for row in delays.tolist():
        acc = torch.zeros((hi - lo, tfb.shape[2]), dtype=torch.int32, device=tfb.device)
        for f, d in enumerate(row):
            s = max_delay - d + lo * ts
            acc += tfb[s:s + (hi - lo) * ts, f].to(torch.int32).view(hi - lo, ts, -1).sum(
                1, dtype=torch.int32)
        out.append((acc.float() / scale).trunc().clamp(-128, 127).to(torch.int8))
    return torch.stack(out, 1)


@pytest.mark.parametrize("F,B", [(6144, 8), (6145, 4), (6500, 12), (6145, 16)])
def test_incoherent_dedispersion_many_channels(cuda, F, B):
    """On either side of the 6144 channels whose row offsets fit a CTA's
    table: beyond, the general kernel reads them from the delays."""
    from skyweaver_b200 import stages
    torch = cuda
    g = np.random.default_rng(F)
    ts, nout, maxd = 2, 21, 15
    delays = _dev(cuda, g.integers(0, maxd + 1, size=(3, F)).astype(np.int32))
    delays[0, 0] = maxd
    tfb = _dev(cuda, g.integers(-128, 128, size=(maxd + nout * ts, F, B)).astype(np.int8))
    got = stages.incoherent_dedisperse(tfb, delays, maxd, ts, 300.0)
    assert torch.equal(got, _idd_rows(torch, tfb, delays, maxd, ts, torch.tensor(300.0, device="cuda"), 0, nout))


@pytest.mark.parametrize("B,gib", [(1024, 33), (1028, 9)])
def test_incoherent_dedispersion_64_bit_offsets(cuda, B, gib):
    """Blocks past 2^31 load units (of 16 and of 4 bytes) keep their row
    offsets in 64 bits: delays that reach from the end of such a block to its
    start, outputs at both ends against plain torch."""
    from skyweaver_b200 import stages
    torch = cuda
    if torch.cuda.mem_get_info()[0] < (gib + 4) << 30:
        pytest.skip("not enough free device memory")
    F, D, ts, nout = 64, 2, 2, 40
    T = (gib << 30) // (F * B)
    maxd = T - nout * ts
    assert T * F * B // (16 if B % 16 == 0 else 4) >= 1 << 31
    tfb = torch.empty((T, F, B), dtype=torch.int8, device="cuda")
    for lo in range(0, T, 4096):
        tfb[lo:lo + 4096].random_(-128, 128)
    delays = torch.linspace(0, maxd, F, device="cuda", dtype=torch.float64).round().to(torch.int32)
    delays = torch.stack([delays, delays.flip(0)])
    got = stages.incoherent_dedisperse(tfb, delays, maxd, ts, 8.0)
    assert torch.equal(got, _idd_rows(torch, tfb, delays, maxd, ts, torch.tensor(8.0, device="cuda"), 0, nout))
