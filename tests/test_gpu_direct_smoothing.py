"""The register-blocked direct convolution (axes that are no power of two)
where its path changes: outputs in eights, pencils in pairs, axes up to 2048
cells, mixed with FFT axes, meshes that start on any float; against the FP64
spectral smoothing."""
import numpy as np
import pytest
import torch

from galaxyfinder_b200 import _lib, batch
from oracle import adjoint as oadj

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda_device):
    c = batch.Context(0)
    yield c
    c.close()


def _desc(nx, ny, nz, cell=0.004, rg=0.008, ptype=5, off=0):
    d = np.zeros(1, _lib.MESH_DTYPE)
    d["nx"], d["ny"], d["nz"], d["ptype"], d["cellsize"], d["rg"], d["off"] = nx, ny, nz, ptype, cell, rg, off
    return d


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a).view(np.uint8)).to("cuda:0")


# The float sums of a pencil round n times: with the kernel's weight in a few
# taps and the roundings independent, sqrt(n) 0.3 u of the result at n = 2049
# is 8e-7 of the largest value; the bar is the mesh path's 2e-6.
@pytest.mark.parametrize("dims", [(3, 5, 7), (9, 11, 15), (17, 36, 37), (100, 6, 33), (63, 65, 129), (130, 64, 9),
                                  (513, 6, 7), (2047, 3, 5), (3, 2047, 5), (5, 3, 2047), (2049, 3, 5), (5, 3, 2049)])
@pytest.mark.parametrize("shift", [0, 1])
def test_direct_lengths(ctx, dims, shift):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx)
    mesh = oadj.Mesh(nx, ny, nz, 0, 0, 0, 0.004, 0.008)
    a = np.zeros((nz, ny, mesh.mx), np.float32)
    a[:, :, :nx] = rng.random((nz, ny, nx)) ** 8
    want = oadj.smooth(a.astype(np.float64), mesh)[:, :, :nx]
    buf = torch.zeros(a.size + 8, dtype=torch.float32, device="cuda:0")
    den = buf[shift:shift + a.size]
    den.copy_(torch.from_numpy(a.ravel()))
    if shift and any(n in (64, 128, 256, 512) for n in dims):
        pytest.skip("FFT axes take meshes as they are planned, on 256-byte boundaries")
    d = _desc(nx, ny, nz)
    _lib.check(_lib.lib().gf_gaussian_smooth(ctx.handle, 1, _lib.ptr(d), _lib.ptr(_dev(d)), _lib.ptr(den)))
    torch.cuda.synchronize()
    got = den.cpu().numpy().reshape(nz, ny, mesh.mx)[:, :, :nx]
    assert np.abs(got - want).max() < 2e-6 * np.abs(want).max()
    assert float(buf[:shift].abs().sum()) == 0 and float(buf[shift + a.size:].abs().sum()) == 0
