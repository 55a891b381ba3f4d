"""Every x / z kernel candidate of the long lines (544 to 2048) and of the 512-long lines, forced in turn (the autotuner
may never pick some of them): x, z convolution, and the one-pass x convolution of a plane, against the register-IO kernels."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LONG = [512, 544, 576, 640, 720, 768, 960, 1024, 1152, 1280, 1536, 2048]


def _run(shape, variant):
    from petakit5d_b200 import _lib, synth
    from petakit5d_b200 import decon as D
    os.environ["PK_TMA_VARIANT"] = str(variant)
    ctx = _lib.Context(0)
    try:
        rng = np.random.default_rng(12)
        vol = np.asfortranarray(rng.integers(90, 3000, size=shape).astype(np.uint16))
        psf = synth.gaussian_psf(tuple(min(9, s) for s in shape), 1.4, 2.5)
        return D.decon_lucy_omw_function(vol, psf, np.asfortranarray(psf[::-1, ::-1, ::-1]), 2, Background=100,
                                         save16bit=False, ctx=ctx)[0].reshape(shape)
    finally:
        ctx.close()
        del os.environ["PK_TMA_VARIANT"]


def _check(shape):
    # the kernels' butterflies differ in rounding only: 2^-24 for each of about 4 operations a stage on a value, log2(4 n)
    # stages at most a transform, and two iterations of two convolutions each (4 transforms of each axis)
    ref = _run(shape, -1)
    tol = 2.0 ** -24 * 4 * np.sqrt(8 * sum(np.log2(4 * n) for n in shape))
    for v in (0, 1, 2):
        J = _run(shape, v)
        err = float(np.linalg.norm((J - ref).ravel()) / np.linalg.norm(ref.ravel()))
        assert err < tol, (shape, v, err, tol)


@pytest.mark.parametrize("n", LONG)
def test_x_lines(n):
    _check((66, n, 9))


@pytest.mark.parametrize("n", LONG)
def test_z_lines(n):
    _check((66, 9, n))


@pytest.mark.parametrize("n", [32, 96, 208, 256, 384] + LONG)
def test_plane_x_convolution(n):
    _check((130, n, 1))
