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
