"""Smoothing of meshes of more than 2^31 cells: the FFT axes along z, whose
last planes lie past 32-bit offsets from a pencil's first cell.  (The other
axes are at the smallest sizes that reach there: 8192 cells by the radix-2
passes, 1030 and 514 by the direct convolution.)

Four unit cells, two of them in the last planes, against the product of the
periodic kernels in FP64.  The bar: the x pass is off by at most 14 u log2(8192)
of a pencil's norm, 1 (see test_gpu_fft_pairs.py), 1.1e-5, which the other two
passes' largest taps, 0.376 each, scale to 1.6e-6; a direct sum of 1030 terms by
1030 u of its value, at most 0.053, 3.3e-6; the z pass by 14 u 9 of the norm of
a column, 0.376^2 times sqrt(2) for a pair, 1.5e-6."""
import numpy as np
import pytest
import torch

from galaxyfinder_b200 import _lib, batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,nz", [(8192, 1030, 256), (8192, 514, 512)])
def test_offsets_past_32_bits(cuda_device, nx, ny, nz):
    mx = 2 * (nx // 2 + 1)
    assert mx * ny * (nz - 1) > 2 ** 31
    cell, rg = 0.004, 0.006
    ctx = batch.Context(0)
    den = torch.zeros((nz, ny, mx), dtype=torch.float32, device=cuda_device)
    units = [(0, 0, 0), (nz // 2, 17, nx - 1), (nz - 1, ny - 1, 4000), (nz - 2, ny // 2, 5001)]
    for u in units:
        den[u] = 1.0
    d = np.zeros(1, _lib.MESH_DTYPE)
    d["nx"], d["ny"], d["nz"], d["ptype"], d["cellsize"], d["rg"] = nx, ny, nz, 5, cell, rg
    _lib.check(_lib.lib().gf_gaussian_smooth(ctx.handle, 1, _lib.ptr(d),
                                             _lib.ptr(torch.from_numpy(d.view(np.uint8)).to(cuda_device)),
                                             _lib.ptr(den)))

    def kernel(n, at):
        k = np.fft.fftfreq(n)
        g = np.exp(-(np.pi * float(np.float32(rg / cell)) * k) ** 2)
        return torch.as_tensor(np.roll(np.fft.ifft(g).real, at), device=cuda_device)

    h = [[kernel(n, a) for n, a in zip((nz, ny, nx), u)] for u in units]
    worst = 0.0
    for k in range(nz):
        want = sum(hz[k] * torch.outer(hy, hx) for hz, hy, hx in h)
        worst = max(worst, float((den[k, :, :nx].double() - want).abs().max()))
    assert worst <= 6.4e-6
    assert float(den[:, :, nx:].abs().max()) == 0.0
    ctx.close()
