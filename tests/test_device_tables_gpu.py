"""A device table whose upload failed is not kept: the next call makes it again.  The failure is the host's: a synchronous
copy is refused while a blocking stream is being captured (cudaErrorStreamCaptureImplicit)."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from petakit5d_b200 import _lib, synth
from petakit5d_b200 import decon as D
from petakit5d_b200 import deskew as DS

pytestmark = pytest.mark.gpu

RELAXED = 2   # cudaStreamCaptureModeRelaxed: allocations go through


class Captured:
    """A blocking stream under capture; the capture is ended and its graph dropped on exit."""

    def __enter__(self):
        self.rt = C.CDLL("libcudart.so.12")
        self.s = C.c_void_p()
        assert self.rt.cudaStreamCreate(C.byref(self.s)) == 0
        assert self.rt.cudaStreamBeginCapture(self.s, RELAXED) == 0
        return self.s.value

    def __exit__(self, *a):
        g = C.c_void_p()
        self.rt.cudaStreamEndCapture(self.s, C.byref(g))   # refused copies have invalidated it
        if g.value:
            self.rt.cudaGraphDestroy(g)
        self.rt.cudaGetLastError()
        self.rt.cudaStreamDestroy(self.s)


def test_erosion_runs():
    shape = (70, 40, 24)
    psf = synth.gaussian_psf((9, 9, 9), 1.2, 2.0)
    psf_b = np.asfortranarray(psf[::-1, ::-1, ::-1])
    vol = synth.puncta_volume(shape, 20, psf, seed=3, background=120.0)
    vol[:30, :10] = 0
    d_in = torch.from_numpy(np.ascontiguousarray(vol.T).view(np.int16)).cuda()
    out = torch.zeros(d_in.shape, dtype=torch.float32, device="cuda")

    def run(ctx, erosion, stream=None):
        D.decon_device("omw", d_in, "uint16", shape, psf, psf_b, 2, ctx=ctx, stream=stream, out=out, Background=100,
                       save16bit=False, EdgeErosion=erosion, deconOffset=0 if erosion else 5.0)

    ctx, fresh = _lib.Context(0), _lib.Context(0)
    try:
        run(ctx, 0)   # tables, OTFs and buffers of the volume (a mask among them) are there
        torch.cuda.synchronize()
        with Captured() as st:
            with pytest.raises(_lib.PkError):
                run(ctx, 4, st)
        run(ctx, 4)
        torch.cuda.synchronize()
        got = out.clone()
        run(fresh, 4)
        torch.cuda.synchronize()
        assert torch.equal(got, out)
    finally:
        ctx.close()
        fresh.close()


def test_skew_slices():
    dims = (48, 40, 30)
    rng = np.random.default_rng(2)
    vol = rng.integers(0, 4000, size=dims[::-1]).astype(np.uint16)
    d_in = torch.from_numpy(vol.view(np.int16)).cuda()
    # a step over xStepThresh: the resampling path with the slice tables
    args = (d_in, "uint16", dims, 32.45, 0.5, 0.108)
    ctx, fresh = _lib.Context(0), _lib.Context(0)
    try:
        od = DS.deskew_rotate_device(*args, save16bit=True, ctx=ctx)
        out = torch.zeros(od[::-1], dtype=torch.int16, device="cuda")
        torch.cuda.synchronize()
        with Captured() as st:
            with pytest.raises(_lib.PkError):
                DS.deskew_rotate_device(*args, out, save16bit=True, ctx=ctx, stream=st)
        DS.deskew_rotate_device(*args, out, save16bit=True, ctx=ctx)
        torch.cuda.synchronize()
        got = out.clone()
        out.zero_()
        torch.cuda.synchronize()
        DS.deskew_rotate_device(*args, out, save16bit=True, ctx=fresh)
        torch.cuda.synchronize()
        assert torch.equal(got, out) and int(out.view(torch.int16).ne(0).sum()) > 0
    finally:
        ctx.close()
        fresh.close()
