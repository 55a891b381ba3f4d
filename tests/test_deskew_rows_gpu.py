"""Deskew / rotate of uint16 rows at the lengths where the row kernels change: whole 16-element blocks, a last group of 8 on
short and long rows, other lengths, and y crops that shift a row's start off its 16-byte groups."""
import numpy as np
import pytest

from oracle import deskew as OD
from petakit5d_b200 import deskew as G

pytestmark = pytest.mark.gpu


def _check(got, ref):
    # the tolerance of the deskew tests: a source coordinate moved across an integer by a rounding step of the 4x4 inverse
    assert got.shape == ref.shape and got.dtype == ref.dtype == np.uint16
    d = np.abs(got.astype(np.int64) - ref.astype(np.int64))
    assert d.max() <= 1 and (d == 0).mean() >= 0.999


@pytest.mark.parametrize("dz,objective", [(0.2, False), (0.65, False), (0.65, True)])   # direct; interpolated; objective scan
@pytest.mark.parametrize("ny", [7, 8, 16, 24, 88, 100, 248, 250, 256, 264, 272, 512, 520])
def test_row_lengths(ny, dz, objective):
    vol = np.asfortranarray(np.random.default_rng(ny).integers(0, 65536, size=(ny, 40, 24)).astype(np.uint16))
    got = G.deskewRotateFrame3D(vol, 32.45, dz, 0.108, save16bit=True, objectiveScan=objective)
    _check(got, OD.deskew_rotate_frame3d(vol, 32.45, dz, 0.108, save16bit=True, objective_scan=objective))


@pytest.mark.parametrize("y0,y1", [(1, 256), (9, 264), (9, 280), (2, 257), (5, 12), (9, 32)])
def test_row_crops(y0, y1):
    vol = np.asfortranarray(np.random.default_rng(y1).integers(0, 65536, size=(288, 40, 24)).astype(np.uint16))
    bbox = (y0, 1, 1, y1, 30, 20)
    got = G.deskewRotateFrame3D(vol, 32.45, 0.65, 0.108, bbox=bbox, save16bit=True)
    _check(got, OD.deskew_rotate_frame3d(vol, 32.45, 0.65, 0.108, bbox=bbox, save16bit=True))
