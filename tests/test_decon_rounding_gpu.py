"""Deconvolutions of lengths without a compile-time plan and of planes, against 64 bits, at the distance that rounding
leaves: a twiddle wrong in its fifth digit shows."""
import math

import numpy as np
import pytest

from oracle import decon as O
from petakit5d_b200 import decon as D
from petakit5d_b200 import synth

pytestmark = pytest.mark.gpu

SHAPES = [(45, 40, 27), (62, 66, 27), (51, 130, 44), (38, 37, 3), (45, 37, 19), (301, 23, 9)]
PLANES = [(66, nx, 1) for nx in (30, 64, 256, 301, 467, 512, 544, 768, 1024, 1280, 2048, 2310)] + [(45, 77, 1), (515, 64, 1)]


@pytest.mark.parametrize("method,numit", [("omw", 2), ("rl", 4)])
@pytest.mark.parametrize("shape", SHAPES + PLANES)
def test_distance_from_64_bits(shape, method, numit):
    psf = synth.gaussian_psf(tuple(min(9, s) for s in shape), 1.2, 2.0)
    psf_b = np.asfortranarray(psf[::-1, ::-1, ::-1]).reshape(psf.shape)
    vol = synth.puncta_volume(shape, 10 + math.prod(shape) // 2000, psf, seed=sum(shape), background=125.0)
    if method == "omw":
        got = D.decon_lucy_omw_function(vol, psf, psf_b, numit, Background=100, save16bit=False)[0]
        ref = O.decon_lucy_omw(vol, psf, psf_b, numit, background=100, save16bit=False, dtype=np.float64)
    else:
        got = D.decon_lucy_function(vol, psf, numit, Background=100, save16bit=False)[0]
        ref = O.decon_lucy(vol, psf, numit, background=100, save16bit=False, dtype=np.float64)
    # 2^-24 for each of about 4 operations a stage on a value, log2(4 n) stages at most a transform, four transforms of
    # each axis an iteration, as a random walk; the ratio's division doubles it, and RL's acceleration
    # (at most the last step once more, and the one before) triples it
    tol = 2.0 ** -24 * 4 * 2 * (3 if method == "rl" else 1) * math.sqrt(4 * numit * sum(math.log2(4 * n) for n in shape))
    assert O.rel_l2(got.reshape(ref.shape), ref) <= tol
