"""Transform lengths without a compile-time plan (gen_engine.cuh, pass_gen.cuh): every radix of the mixed-radix
engine, lengths with a larger prime factor (stage_direct), and those that keep the plain in-place engine."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import decon as O
from petakit5d_b200 import decon as D
from petakit5d_b200 import synth

pytestmark = pytest.mark.gpu

# x / z lengths: primes of the radix set, composites of one and several stages, larger primes alone and beside
# register radices on tiles of 32 to 4 columns, one and several TMA boxes a line, and lengths above 2048 with
# a large prime (the plain in-place engine)
LENGTHS = [3, 6, 7, 11, 13, 15, 17, 19, 22, 23, 27, 29, 31, 33, 37, 62, 97, 122, 130, 251, 257, 270, 299, 467, 520, 521,
           613, 930, 1140, 1151, 1558, 1721, 2047, 2310, 3001, 4093]


def _tol(dims):
    # a transform's rounding grows with its stages: 2^-24 for each of about 4 operations on a value
    # per stage, log2(4 n) stages at most, twice (plain sums over a prime factor round p times each)
    return 2.0 ** -24 * 4 * sum(math.log2(4 * n) + (math.log2(4 * n) if n > 1 else 0) for n in dims)


def _roundtrip(ny, nx, nz):
    g = torch.Generator(device="cuda").manual_seed(ny * 7919 + nx * 31 + nz)
    x = torch.rand((nz, nx, ny), generator=g, device="cuda") - 0.5
    py = ny // 2 + 1
    S = torch.zeros((nz, nx, py), dtype=torch.complex64, device="cuda")
    back = torch.zeros_like(x)
    torch.cuda.synchronize()
    D.fft3_r2c(x, (ny, nx, nz), S)
    torch.cuda.synchronize()
    ref = torch.fft.rfftn(x.double())
    tol = _tol((ny, nx, nz))
    assert float((S - ref).norm() / ref.norm()) <= tol
    D.fft3_c2r(S, (ny, nx, nz), back)
    torch.cuda.synchronize()
    n = ny * nx * nz
    assert float((back.double() / n - x.double()).norm() / x.double().norm()) <= 2 * tol


@pytest.mark.parametrize("n", LENGTHS)
def test_x_lengths(n):
    _roundtrip(34, n, 3)


@pytest.mark.parametrize("n", LENGTHS)
def test_z_lengths(n):
    _roundtrip(16, 5, n)


@pytest.mark.parametrize("ny", [3, 7, 9, 25, 37, 38, 74, 97, 194, 251, 301, 302, 467, 602, 934, 1001, 1140, 1531, 2047,
                                3062, 4093, 8186])
def test_y_lengths(ny):
    _roundtrip(ny, 5, 3)


@pytest.mark.parametrize("method,numit", [("omw", 2), ("rl", 5)])
@pytest.mark.parametrize("shape", [(45, 37, 19), (62, 66, 27), (51, 130, 41), (38, 37, 3)])
def test_decon_matches_oracle(shape, method, numit):
    psf = synth.gaussian_psf(tuple(min(9, s) for s in shape), 1.2, 2.0)
    vol = synth.puncta_volume(shape, 60, psf, seed=sum(shape), background=120.0)
    kw = dict(Background=100, save16bit=False)
    if method == "omw":
        got = D.decon_lucy_omw_function(vol, psf, psf[::-1, ::-1, ::-1], numit, **kw)[0]
        ref = O.decon_lucy_omw(vol, psf, psf[::-1, ::-1, ::-1], numit, background=100, save16bit=False, dtype=np.float64)
    else:
        got = D.decon_lucy_function(vol, psf, numit, **kw)[0]
        ref = O.decon_lucy(vol, psf, numit, background=100, save16bit=False, dtype=np.float64)
    # the repository's tolerances: 1e-4 for two OMW iterations, 1e-3 for RL
    assert O.rel_l2(got, ref) <= (1e-4 if method == "omw" else 1e-3)
