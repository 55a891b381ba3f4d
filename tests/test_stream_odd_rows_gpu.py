"""Single-precision frames with odd rows: the streamed host call equals the device call bit for bit.  Odd rows run in pairs,
and slabs begin at any plane: with odd nx a slab's first row could be the second of a pair of the whole volume."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from petakit5d_b200 import _lib
from petakit5d_b200 import decon as D
from petakit5d_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method,numit", [("omw", 2), ("rl", 3)])
@pytest.mark.parametrize("shape", [(45, 33, 63), (105, 39, 49), (45, 34, 63)])
def test_streamed_host_call_equals_device_call(shape, method, numit):
    psf = synth.gaussian_psf((9, 9, 9), 1.3, 2.0)
    vol = np.asfortranarray(synth.puncta_volume(shape, 40, psf, seed=3, background=120.0).astype(np.float32))
    psf_b = np.asfortranarray(psf[::-1, ::-1, ::-1])
    ctx = _lib.Context(0)
    try:
        kw = dict(Background=100, save16bit=False)
        if method == "omw":
            got = D.decon_lucy_omw_function(vol, psf, psf_b, numit, ctx=ctx, **kw)[0]
        else:
            got = D.decon_lucy_function(vol, psf, numit, ctx=ctx, **kw)[0]
        d_in = torch.from_numpy(np.ascontiguousarray(vol.T)).cuda()
        d_out = torch.empty_like(d_in)
        D.decon_device(method, d_in, "float32", shape, psf, psf_b if method == "omw" else None, numit, out=d_out, ctx=ctx, **kw)
        torch.cuda.synchronize()
        assert np.array_equal(got, d_out.cpu().numpy().T)
    finally:
        ctx.close()
