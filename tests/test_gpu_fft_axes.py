"""The register transforms of 64-, 128- and 256-cell axes (and the 512-cell
Stockham passes) on tiles with every kind of remainder: one pencil, odd counts,
one more and one less than a tile, along each axis; against the FP64 spectral
smoothing at the smoothing's bar (log2(n) <= 9 stages of float roundings stay
below 2e-6 of the mesh's largest value)."""
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


@pytest.mark.parametrize("n", [64, 128, 256, 512])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("other", [(1, 1), (1, 3), (3, 11), (31, 1), (32, 2), (33, 3), (65, 1)])
def test_tile_remainders(ctx, n, axis, other):
    dims = list(other)
    dims.insert(axis, n)
    nx, ny, nz = dims
    rng = np.random.default_rng(n + axis)
    mesh = oadj.Mesh(nx, ny, nz, 0, 0, 0, 0.004, 0.007)
    a = np.zeros((nz, ny, mesh.mx), np.float32)
    a[:, :, :nx] = rng.random((nz, ny, nx)) ** 8
    want = oadj.smooth(a.astype(np.float64), mesh)[:, :, :nx]
    d = np.zeros(1, _lib.MESH_DTYPE)
    d["nx"], d["ny"], d["nz"], d["ptype"], d["cellsize"], d["rg"] = nx, ny, nz, 5, 0.004, 0.007
    den = torch.from_numpy(a.ravel()).to("cuda:0")
    _lib.check(_lib.lib().gf_gaussian_smooth(ctx.handle, 1, _lib.ptr(d),
                                             _lib.ptr(torch.from_numpy(d.view(np.uint8)).to("cuda:0")), _lib.ptr(den)))
    torch.cuda.synchronize()
    got = den.cpu().numpy().reshape(nz, ny, mesh.mx)
    assert np.abs(got[:, :, :nx] - want).max() < 2e-6 * np.abs(want).max()
    assert np.array_equal(got[:, :, nx:], a[:, :, nx:])  # the row padding is not touched
