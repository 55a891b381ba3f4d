"""One-plane volumes convolve in one x pass (forward, OTF, inverse on the tile): every kernel family against the
oracle -- short plans (register-IO, TMA), 512 to 2048 lines, lengths without a plan, a large prime, a lone column."""
import numpy as np
import pytest

from oracle import decon as O
from petakit5d_b200 import decon as D
from petakit5d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx", [1, 2, 30, 64, 256, 301, 467, 512, 544, 768, 1024, 1280, 2048, 2310])
@pytest.mark.parametrize("method,numit", [("omw", 2), ("rl", 4)])
def test_plane_matches_oracle(nx, method, numit):
    shape = (66, nx, 1)
    psf = synth.gaussian_psf((9, min(9, nx), 1), 1.3, 1.0)
    vol = synth.puncta_volume(shape, 5 + nx // 8, psf, seed=nx, background=130.0)
    if method == "omw":
        got = D.decon_lucy_omw_function(vol, psf, psf[::-1, ::-1], numit, Background=100, save16bit=False)[0]
        ref = O.decon_lucy_omw(vol, psf, psf[::-1, ::-1], numit, background=100, save16bit=False, dtype=np.float64)
    else:
        got = D.decon_lucy_function(vol, psf, numit, Background=100, save16bit=False)[0]
        ref = O.decon_lucy(vol, psf, numit, background=100, save16bit=False, dtype=np.float64)
    # the repository's tolerances: 1e-4 for two OMW iterations, 1e-3 for RL
    assert O.rel_l2(got.reshape(ref.shape), ref) <= (1e-4 if method == "omw" else 1e-3)
