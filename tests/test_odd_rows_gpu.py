"""Odd row lengths run two rows as one complex transform: a row must not see its partner."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from petakit5d_b200 import decon as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny", [9, 45, 95, 1001])
def test_c2r_of_a_spectrum_without_symmetry(ny):
    # the inverse along y takes the real part of bin 0, as irfft does, whatever its imaginary part
    nx, nz = 5, 3
    g = torch.Generator(device="cuda").manual_seed(ny)
    S = torch.randn((nz, nx, ny // 2 + 1), generator=g, device="cuda", dtype=torch.complex64)
    out = torch.zeros((nz, nx, ny), device="cuda")
    torch.cuda.synchronize()
    D.fft3_c2r(S.clone(), (ny, nx, nz), out)
    torch.cuda.synchronize()
    ref = torch.fft.irfft(torch.fft.ifft2(S.to(torch.complex128), dim=(0, 1)), n=ny, dim=2) * (ny * nx * nz)
    # 2^-24 for each of about 4 operations a stage on a value, at most log2(4 n) stages an axis, forward errors in norm
    tol = 2.0 ** -24 * 8 * (np.log2(4 * ny) + np.log2(4 * nx) + np.log2(4 * nz))
    assert float((out.double() - ref).norm() / ref.norm()) <= tol
