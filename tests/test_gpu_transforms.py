"""The line transforms of the shift search and the Fourier shift at the lengths
where their index arithmetic changes (shortest and longest lines, odd heights,
every radix, powers of two beside other lengths), against NumPy's FP64 FFT.

Tolerance: a transform pass rounds each point a few times (about 2 x 2^-24
relative, uncorrelated or not); the longest case runs 3 transforms per axis of
at most 8 passes, 24 passes x 2 x 2^-24 = 2.9e-6, rounded up."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 3e-6


def rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("ny,nx", [(2, 2), (3, 16), (15, 32), (16, 4096), (4096, 16), (9, 4000),
                                   (125, 1024), (2187, 2), (7, 8), (63, 2401), (1050, 64)])
def test_correlation_image(gb, ny, nx):
    import torch

    rng = np.random.default_rng(ny * 5000 + nx)
    a, b = rng.standard_normal((2, ny, nx)).astype(np.float32)
    A, B = np.fft.fft2(a.astype(np.float64)), np.fft.fft2(b.astype(np.float64))
    ref = np.fft.ifft2(np.conj(A) * B).real * (nx * ny)
    c = torch.zeros(ny, nx, device="cuda")
    gb.ccorr2d_device(torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda(), c)
    assert rel(c.cpu().numpy(), ref) < TOL


@pytest.mark.parametrize("nz,ny,nx", [(1, 2, 2), (2, 3, 16), (2, 16, 3), (3, 15, 32), (1, 2, 4096),
                                      (1, 2048, 16), (2, 6, 10), (2, 189, 250), (1, 1, 8)])
def test_fourier_shift(gb, nz, ny, nx):
    import torch

    rng = np.random.default_rng(ny * 5000 + nx)
    a = rng.standard_normal((nz, ny, nx)).astype(np.float32)
    s = rng.uniform(-20, 20, (2, nz)).astype(np.float32)
    out = torch.zeros(nz, ny, nx, device="cuda")
    args = (torch.from_numpy(a).cuda(), out, torch.from_numpy(s[0]).cuda(),
            torch.from_numpy(s[1]).cuda())
    if ny < 2:
        with pytest.raises(RuntimeError):
            gb.fshift2d_device(*args)
        return
    gb.fshift2d_device(*args)
    ky, kx = np.fft.fftfreq(ny)[:, None], np.fft.fftfreq(nx)[None, :]
    for z in range(nz):
        ph = np.exp(-2j * np.pi * (float(s[0, z]) * kx + float(s[1, z]) * ky))
        ref = np.fft.ifft2(np.fft.fft2(a[z].astype(np.float64)) * ph).real
        assert rel(out[z].cpu().numpy(), ref) < TOL
