"""Row lengths with a prime factor above 31 beside a register radix, too long for the tiles of the register-tiled sums:
they run on the plain in-place engine."""
import math

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import decon as O
from petakit5d_b200 import decon as D
from petakit5d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [515, 519, 555, 999, 1036, 1110, 1332, 2452])
@pytest.mark.parametrize("nx,nz", [(5, 3), (34, 7)])
def test_round_trip(ny, nx, nz):
    # rows of several tiles, an odd number of them in the first case
    g = torch.Generator(device="cuda").manual_seed(ny + nx)
    x = torch.rand((nz, nx, ny), generator=g, device="cuda") - 0.5
    S = torch.zeros((nz, nx, ny // 2 + 1), dtype=torch.complex64, device="cuda")
    back = torch.zeros_like(x)
    torch.cuda.synchronize()
    D.fft3_r2c(x, (ny, nx, nz), S)
    torch.cuda.synchronize()
    ref = torch.fft.rfftn(x.double())
    # 2^-24 for each of about 4 operations on a value per stage, log2(4 n) stages at most an axis, twice (a plain sum
    # over a prime factor rounds as often as it has terms, as a random walk)
    tol = 2.0 ** -24 * 8 * sum(math.log2(4 * n) for n in (ny, nx, nz))
    assert float((S - ref).norm() / ref.norm()) <= tol
    D.fft3_c2r(S, (ny, nx, nz), back)
    torch.cuda.synchronize()
    assert float((back.double() / (ny * nx * nz) - x.double()).norm() / x.double().norm()) <= 2 * tol


@pytest.mark.parametrize("method,numit", [("omw", 2), ("rl", 4)])
@pytest.mark.parametrize("shape", [(515, 20, 9), (1036, 13, 6), (999, 34, 1)])
def test_decon_matches_oracle(shape, method, numit):
    psf = synth.gaussian_psf(tuple(min(9, s) for s in shape), 1.2, 2.0)
    psf_b = np.asfortranarray(psf[::-1, ::-1, ::-1]).reshape(psf.shape)
    vol = synth.puncta_volume(shape, 60, psf, seed=sum(shape), background=120.0)
    if method == "omw":
        got = D.decon_lucy_omw_function(vol, psf, psf_b, numit, Background=100, save16bit=False)[0]
        ref = O.decon_lucy_omw(vol, psf, psf_b, numit, background=100, save16bit=False, dtype=np.float64)
    else:
        got = D.decon_lucy_function(vol, psf, numit, Background=100, save16bit=False)[0]
        ref = O.decon_lucy(vol, psf, numit, background=100, save16bit=False, dtype=np.float64)
    # a transform's error by the bound above, 8 transforms of each axis an iteration, as a random walk; dark voxels'
    # ratios take it up once more
    tol = 2.0 ** -24 * 8 * sum(math.log2(4 * n) for n in shape) * math.sqrt(8 * numit)
    assert O.rel_l2(got.reshape(ref.shape), ref) <= tol
