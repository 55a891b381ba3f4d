"""Edge erosion on packed words (k_mask_pack / k_mask_disk / k_mask_line): exact against the oracle at word
edges, runs of several words, planes, full masks, and through the deconvolution's mask options."""
import numpy as np
import pytest
from scipy import ndimage

from oracle import decon as O
from petakit5d_b200 import decon as D
from petakit5d_b200 import synth

pytestmark = pytest.mark.gpu


def _ref(mask, E):
    """oracle.decon.mask_edge_erosion, with scipy's erosion (outside counts as set) so that the neighbourhood
    may be larger than the volume."""
    if mask.all():
        return O.mask_edge_erosion(mask, E)
    m = mask.copy()
    flat = m.shape[2] == 1
    for ax in range(2 if flat else 3):
        idx = [slice(None)] * 3
        idx[ax] = [0, -1]
        m[tuple(idx)] = False
    m = ndimage.binary_erosion(m, structure=O.disk_nhood(E - 1)[:, :, None], border_value=1)
    return m if flat else ndimage.binary_erosion(m, structure=np.ones((1, 1, 2 * E - 1), bool), border_value=1)


@pytest.mark.parametrize("E", [1, 2, 3, 5, 8, 32, 33, 40])
@pytest.mark.parametrize("shape", [(31, 7, 5), (32, 9, 1), (33, 40, 3), (64, 33, 6), (97, 50, 17), (1100, 5, 3)])
def test_mask_matches_oracle(shape, E):
    rng = np.random.default_rng(E * 1000 + sum(shape))
    m = np.ones(shape, bool)
    idx = rng.integers(0, m.size, size=max(1, m.size // 4000))
    m.ravel()[idx] = False
    m[: shape[0] // 5] = False
    assert np.array_equal(D.decon_mask_edge_erosion(m, E), _ref(m, E))
    full = np.ones(shape, bool)
    assert np.array_equal(D.decon_mask_edge_erosion(full, E), O.mask_edge_erosion(full, E))


@pytest.mark.parametrize("zeros", [False, True])
@pytest.mark.parametrize("ny", [64, 512])
def test_decon_with_erosion_offset_and_scale(ny, zeros):
    shape = (ny, 20, 9)
    psf = synth.gaussian_psf((7, 7, 5), 1.2, 1.5)
    vol = synth.puncta_volume(shape, 40, psf, seed=ny, background=120.0)
    if zeros:
        vol[:9, :, 2:5] = 0
    for save16 in (False, True):
        kw = dict(background=100, scale=1.5, offset=3.0, edge_erosion=3, save16bit=save16)
        ref = O.decon_lucy_omw(vol, psf, psf[::-1, ::-1, ::-1], 2, dtype=np.float32, **kw)
        got = D.decon_lucy_omw_function(vol, psf, psf[::-1, ::-1, ::-1], 2, Background=100, scaleFactor=1.5, deconOffset=3.0,
                                        EdgeErosion=3, save16bit=save16)[0]
        assert np.array_equal(got == 0, ref == 0)
        if save16:
            assert int(np.max(np.abs(got.astype(int) - ref.astype(int)))) <= 1
        else:
            assert O.rel_l2(got, ref) <= 1e-4
