"""pk_decon_lucy_omw_noalloc runs the engines of the plain call: at lengths without a compile-time plan (mixed radices up
to 16 and above, a large prime factor) and for volumes of one plane its results equal pk_decon_lucy_omw_device's bit for bit."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from petakit5d_b200 import _lib, synth

pytestmark = pytest.mark.gpu


def _run(fn, shape, vol, psf, psf_b):
    p = _lib.DeconParams()
    _lib.lib.pk_params_default(p)
    p.background = 100.0
    p.save16bit = 0
    d_in = torch.from_numpy(np.ascontiguousarray(vol.T).view(np.int16)).cuda()
    out = torch.empty(d_in.shape, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    args = (d_in.data_ptr(), _lib.PK_U16, _lib.i64x3(shape), psf.ctypes.data, _lib.i64x3(psf.shape), psf_b.ctypes.data,
            _lib.i64x3(psf_b.shape), 2, p, out.data_ptr(), torch.cuda.current_stream().cuda_stream)
    _lib.check(fn(*args))
    torch.cuda.synchronize()
    return out.cpu().numpy().T


@pytest.mark.parametrize("shape", [(62, 40, 27), (45, 38, 27), (45, 37, 19), (74, 40, 15), (130, 66, 1), (45, 37, 1),
                                   (130, 38, 70), (1, 40, 27), (6, 1, 1)])
def test_noalloc_equals_device_call(shape, monkeypatch):
    monkeypatch.setenv("PK_TMA_VARIANT", "-1")   # the no-allocation call runs the register-IO kernels where a plan exists
    psf = synth.gaussian_psf(tuple(min(9, s) for s in shape), 1.3, 2.0)
    psf = np.asfortranarray(psf, np.float32).reshape(tuple(min(9, s) for s in shape), order="F")
    psf_b = np.asfortranarray(psf[::-1, ::-1, ::-1])
    vol = np.asfortranarray(synth.puncta_volume(shape, 10, psf, seed=9, background=110.0).reshape(shape, order="F"))
    ctx = _lib.default_context()
    got = _run(lambda *a: _lib.lib.pk_decon_lucy_omw_noalloc(*a), shape, vol, psf, psf_b)
    ref = _run(lambda *a: _lib.lib.pk_decon_lucy_omw_device(ctx.handle, *a), shape, vol, psf, psf_b)
    assert np.array_equal(got, ref)
