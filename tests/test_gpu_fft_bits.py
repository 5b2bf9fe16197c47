"""The smoothing's register transforms give the bits of Stockham passes of radix
8, 8 and n / 64 through shared memory, which they replaced: sha256 of the smoothed
meshes, as those passes left them on these inputs.  (A mesh density's gradient is
the difference of sums over a mesh; what its roundings are decides its last
digits.)  The other two axes have lengths of 1 and 32, a direct and a radix-2 axis
without a choice of roundings."""
import hashlib

import numpy as np
import pytest
import torch

from galaxyfinder_b200 import _lib, batch

pytestmark = pytest.mark.gpu

DIGESTS = {
    (64, 32, 1, 0): "9bd432c7882063d36526c2f7",
    (64, 32, 1, 1): "2e1c7172072c0449367d3dc7",
    (1, 64, 32, 0): "2109e13c56d678f92e406faf",
    (1, 64, 32, 1): "ef31b1dc5cd5543b4b062b7f",
    (32, 1, 64, 0): "4a2f4663858c619c0f4cc6ea",
    (32, 1, 64, 1): "d3a02cc44f669cc48873d6cf",
    (128, 32, 1, 0): "3ab60cb3e8c303c300df0d48",
    (128, 32, 1, 1): "1ed0cbbe44d623c20733080c",
    (1, 128, 32, 0): "f2198495f928e4d9ceb2c94d",
    (1, 128, 32, 1): "7e50c1628e9461dc4863a303",
    (32, 1, 128, 0): "b1bc767820910507221b728f",
    (32, 1, 128, 1): "798db9d5d14e003810d31042",
    (256, 32, 1, 0): "14edf6a2595a1a27d97207e0",
    (256, 32, 1, 1): "d633d94f97c586d52541e710",
    (1, 256, 32, 0): "8044372f8efd2d4126d54406",
    (1, 256, 32, 1): "b072319529740bebe17a9eee",
    (32, 1, 256, 0): "4d79fcd767483931a7539ae1",
    (32, 1, 256, 1): "821f072811bf9126ad6fb083",
    (64, 128, 256, 0): "d7a8c74706c8f1e38eb47699",
    (256, 64, 64, 1): "1f014a16a878d2b657af89a8",
}


def smoothed(ctx, dims, kind):
    """A mesh of eighth powers (0) or of sparse values over six decades (1)."""
    nx, ny, nz = dims
    mx = 2 * (nx // 2 + 1)
    rng = np.random.default_rng(nx + 3 * ny + 5 * nz + kind)
    a = rng.random((nz, ny, mx)) ** 8
    if kind:
        a = np.where(rng.random(a.shape) < 0.03, 10.0 ** (6.0 * a), 0.0)
    a = a.astype(np.float32)
    d = np.zeros(1, _lib.MESH_DTYPE)
    d["nx"], d["ny"], d["nz"], d["ptype"], d["cellsize"], d["rg"] = nx, ny, nz, 5, 0.004, 0.006
    den = torch.from_numpy(a.ravel()).to("cuda:0")
    _lib.check(_lib.lib().gf_gaussian_smooth(ctx.handle, 1, _lib.ptr(d),
                                             _lib.ptr(torch.from_numpy(d.view(np.uint8)).to("cuda:0")), _lib.ptr(den)))
    torch.cuda.synchronize()
    return np.ascontiguousarray(den.cpu().numpy().reshape(a.shape)[:, :, :nx])


CASES = [(*(n if i == axis else (32 if i == (axis + 1) % 3 else 1) for i in range(3)), kind)
         for n in (64, 128, 256) for axis in range(3) for kind in (0, 1)] + [(64, 128, 256, 0), (256, 64, 64, 1)]


@pytest.mark.parametrize("nx,ny,nz,kind", CASES)
def test_bits_of_the_stockham_passes(cuda_device, nx, ny, nz, kind):
    ctx = batch.Context(0)
    got = smoothed(ctx, (nx, ny, nz), kind)
    ctx.close()
    assert hashlib.sha256(got.tobytes()).hexdigest()[:24] == DIGESTS[nx, ny, nz, kind]
