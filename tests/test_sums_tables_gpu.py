"""Root matrices of lengths with a prime factor above 31: a context keeps a bounded amount, gives them back on reset, and
where it keeps none the plain engine forms the same sums."""
import ctypes as C
import json

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from petakit5d_b200 import _lib, synth
from petakit5d_b200 import decon as D

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _decon(method, shape, ctx, numit=2):
    psf = synth.gaussian_psf(tuple(min(9, s) for s in shape), 1.2, 2.0)
    vol = synth.puncta_volume(shape, 20, psf, seed=sum(shape), background=120.0)
    if method == "omw":
        psf_b = np.asfortranarray(psf[::-1, ::-1, ::-1]).reshape(psf.shape)
        return D.decon_lucy_omw_function(vol, psf, psf_b, numit, Background=100, save16bit=False, ctx=ctx)[0]
    return D.decon_lucy_function(vol, psf, numit, Background=100, save16bit=False, ctx=ctx)[0]


def _free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


# tiles of 32, 16, 8 and 4 lines, whole and partly filled, lengths of one and of several prime factors, on each axis
SHAPES = [(82, 41, 38), (130, 37, 43), (70, 233, 3), (129, 467, 5), (140, 613, 2), (6, 467, 60), (26, 101, 40), (118, 74, 6),
          (202, 9, 5), (222, 66, 5), (301, 9, 5), (74, 1, 40), (66, 74, 1), (467, 3, 2)]


def _engines(shape):
    buf = C.create_string_buffer(4096)
    assert _lib.lib.pk_plan_read(_lib.i64x3(shape), buf, len(buf)) > 0
    return [a["engine"] for a in json.loads(buf.value)]


@pytest.mark.parametrize("method,numit", [("omw", 2), ("rl", 4)])
@pytest.mark.parametrize("shape", SHAPES)
def test_same_results_without_the_matrices(shape, method, numit, monkeypatch):
    assert "sums" in _engines(shape)
    ctx = _lib.Context(0)
    ref = _decon(method, shape, ctx, numit)
    ctx.close()
    monkeypatch.setenv("PK_SUMS_MB", "0")
    ctx = _lib.Context(0)
    try:
        for _ in range(2):
            assert np.array_equal(_decon(method, shape, ctx, numit), ref)
    finally:
        ctx.close()


def test_bounded(monkeypatch):
    # a prime near 1030 has 8.5 MB of matrices: 12 lengths would take 100 MB
    monkeypatch.setenv("PK_SUMS_MB", "20")
    ctx = _lib.Context(0)
    try:
        _decon("omw", (16, 1009, 2), ctx)
        before = _free()
        for n in (1013, 1019, 1021, 1031, 1033, 1039, 1049, 1051, 1061, 1063, 1069):
            _decon("omw", (16, n, 2), ctx)
        # the second length's matrices, and room for the volumes' spectra, twiddles and programs (under 1 MB a length)
        assert before - _free() <= 24 * MB
    finally:
        ctx.close()


def test_reset_gives_them_back():
    ctx = _lib.Context(0)
    try:
        for n in (1987, 1993, 1997, 1999):   # 32 MB each
            _decon("omw", (16, n, 2), ctx)
        before = _free()
        _lib.check(_lib.lib.pk_ctx_reset(ctx.handle))
        assert _free() - before >= 4 * 30 * MB
        _decon("omw", (16, 1999, 2), ctx)
    finally:
        ctx.close()
