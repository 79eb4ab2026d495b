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
