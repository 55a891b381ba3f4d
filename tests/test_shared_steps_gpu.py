"""A volume's result does not depend on the volumes that share its launches: batches and served mixes of volumes on
different transform engines (plain sums beside mixed radices, radices up to 16 beside larger ones) and of planes beside
volumes equal the single calls bit for bit."""
import numpy as np
import pytest

from petakit5d_b200 import chunking as K
from petakit5d_b200 import decon as D
from petakit5d_b200 import serve as SV
from petakit5d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def register_io(monkeypatch):
    # lengths with a plan: one kernel for single and shared launches, whatever the autotuner would pick for each
    monkeypatch.setenv("PK_TMA_VARIANT", "-1")


def _volumes(shapes):
    psf = synth.gaussian_psf((9, 9, 7), 1.3, 1.6)
    return psf, [synth.puncta_volume(s, 20, _psf(psf, s), seed=40 + i, background=100.0) for i, s in enumerate(shapes)]


def _psf(psf, shape):
    return np.asfortranarray(psf[:, :, 3:4]) if shape[2] == 1 else psf


def _alone(method, vol, psf, numit):
    if method == "omw":
        return D.decon_lucy_omw_function(vol, psf, psf[::-1, ::-1, ::-1], numit, Background=100, save16bit=False)[0]
    return D.decon_lucy_function(vol, psf, numit, Background=100, save16bit=False)[0]


def _batch(method, vols, psf, numit):
    psfs = [psf, np.asfortranarray(psf[:, :, 3:4])]
    ids = [1 if v.shape[2] == 1 else 0 for v in vols]
    psfs_b = [np.asfortranarray(p[::-1, ::-1, ::-1]) for p in psfs] if method == "omw" else None
    return K.batch_decon(vols, psfs, ids, numit, method, psfs_b, None, Background=100, save16bit=False)


# z 40 and x 40 run the mixed-radix engine, beside a prime above 31 the plain sums; x 38 has a radix above 16; a volume
# of one plane convolves in one x pass
MIXES = [
    [(64, 37, 40), (64, 40, 40), (64, 41, 40), (64, 42, 40)],
    [(64, 40, 40), (64, 40, 37), (74, 40, 40)],
    [(62, 38, 27), (62, 40, 27), (45, 38, 27), (45, 40, 27)],
    [(64, 40, 1), (64, 40, 20), (64, 42, 1), (64, 40, 20)],
    [(64, 64, 1), (64, 64, 32), (64, 37, 1), (64, 512, 1)],
]


@pytest.mark.parametrize("method,numit", [("omw", 2), ("rl", 4)])
@pytest.mark.parametrize("shapes", MIXES, ids=str)
def test_batch_equals_single_calls(shapes, method, numit):
    psf, vols = _volumes(shapes)
    for v, o in zip(vols, _batch(method, vols, psf, numit)):
        assert np.array_equal(o.reshape(v.shape), _alone(method, v, _psf(psf, v.shape), numit).reshape(v.shape)), v.shape


@pytest.mark.parametrize("device_loop", [False, True])
@pytest.mark.parametrize("shapes", MIXES, ids=str)
def test_served_equals_single_calls(shapes, device_loop):
    psf, vols = _volumes(shapes)
    with SV.Server(budget_bytes=4e9, max_batch=8, device_loop=device_loop) as srv:
        for i, p in enumerate([psf, np.asfortranarray(psf[:, :, 3:4])]):
            srv.add_psf(i, p, np.asfortranarray(p[::-1, ::-1, ::-1]))
        ids = [srv.submit(v, 1 if v.shape[2] == 1 else 0, m, n, Background=100, save16bit=False)
               for v in vols for m, n in (("omw", 2), ("rl", 4))]
        outs = [srv.wait(i)[0] for i in ids]
    for k, o in enumerate(outs):
        v = vols[k // 2]
        m, n = (("omw", 2), ("rl", 4))[k % 2]
        assert np.array_equal(o.reshape(v.shape), _alone(m, v, _psf(psf, v.shape), n).reshape(v.shape)), (v.shape, m)
