"""The vector reductions of the scattered mesh deposits (three cells of a row
across 8- and 16-byte words): meshes that start on any float, rows of every
alignment, stencils at the ends of the mesh, nothing written outside it."""
import ctypes

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


def _particles(rng, n, dims, cell):
    """Positions over the whole mesh, the outermost stencils among them."""
    hi = np.array(dims) - 2.0
    g = 1.0 + rng.random((n, 3)) * (hi - 1.0)
    g[:8] = [[1 if b & 1 else hi[0], 1 if b & 2 else hi[1], 1 if b & 4 else hi[2]] for b in range(8)]
    return g * cell


@pytest.mark.parametrize("dims", [(16, 9, 8), (17, 8, 9), (18, 7, 7), (31, 6, 5), (4, 4, 4)])
@pytest.mark.parametrize("shift", [0, 1, 2, 3, 4])
def test_deposit_alignments(ctx, restatement, dims, shift):
    nx, ny, nz = dims
    rng = np.random.default_rng(nx + 100 * shift)
    n, cell = 3000, 0.004
    p = _particles(rng, n, dims, cell)
    m = 10 ** rng.uniform(6, 8, n)
    db = batch.DeviceBatch.from_arrays(p[:, 0], p[:, 1], p[:, 2], m, np.full(n, 2), [0, n])
    total = 2 * (nx // 2 + 1) * ny * nz
    buf = torch.full((total + 16,), 7.5, dtype=torch.float32, device="cuda:0")
    den = buf[shift:shift + total]
    d = _desc(nx, ny, nz)
    b = db.c()
    _lib.check(_lib.lib().gf_tsc_deposit(ctx.handle, ctypes.byref(b), _lib.ptr(_dev(d)), _lib.ptr(d), _lib.ptr(den)))
    torch.cuda.synchronize()
    want = restatement.tsc(p[:, 0], p[:, 1], p[:, 2], m, np.full(n, 2, np.int32), nx, ny, nz, 0, 0, 0, cell, 5,
                           acc_double=True)
    got = den.cpu().numpy()
    # the stencil values are the same floats; t positive terms summed in any
    # order lie within t u of their exact sum
    i0, j0, k0, *_ = oadj._stencil(p, oadj.Mesh(nx, ny, nz, 0, 0, 0, cell, 0.008))
    t = np.zeros((nz, ny, 2 * (nx // 2 + 1)))
    for c in range(3):
        for b in range(3):
            for a in range(3):
                np.add.at(t, (k0 + c, j0 + b, i0 + a), 1)
    assert np.all(np.abs(got - want) <= (t.ravel() + 1) * 2.0 ** -24 * want)
    assert bool((buf[:shift] == 7.5).all()) and bool((buf[shift + total:] == 7.5).all())


@pytest.mark.parametrize("nx", [16, 17, 18])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_mesh_gradient_alignments(ctx, nx, shift):
    ny, nz, n, cell = 9, 8, 2000, 0.004
    rng = np.random.default_rng(nx + shift)
    p = _particles(rng, n, (nx, ny, nz), cell)
    g = rng.standard_normal(n)
    db = batch.DeviceBatch.from_arrays(p[:, 0], p[:, 1], p[:, 2], np.ones(n), np.full(n, 2), [0, n])
    total = 2 * (nx // 2 + 1) * ny * nz
    buf = torch.zeros(total + 16, dtype=torch.float32, device="cuda:0")
    gs = buf[shift:shift + total]
    S = torch.from_numpy(rng.random(total).astype(np.float32)).to("cuda:0")
    gx, gy, gz = (torch.zeros(n, dtype=torch.float64, device="cuda:0") for _ in range(3))
    gd = torch.from_numpy(g).to("cuda:0")
    d = _desc(nx, ny, nz)
    b = db.c()
    _lib.check(_lib.lib().gf_find_den_adjoint(ctx.handle, ctypes.byref(b), _lib.ptr(_dev(d)), _lib.ptr(S), _lib.ptr(gd),
                                              _lib.ptr(gs), _lib.ptr(gx), _lib.ptr(gy), _lib.ptr(gz)))
    torch.cuda.synchronize()
    mesh = oadj.Mesh(nx, ny, nz, 0, 0, 0, cell, 0.008)
    gp, want = oadj.find_den_grad(p, S.cpu().numpy(), mesh, g)
    # up to 200 signed float terms per cell of size |g| W < 1.7
    assert np.abs(gs.cpu().numpy() - want.ravel()).max() < 200 * 2.0 ** -24 * 1.7 * 4
    np.testing.assert_allclose(torch.stack([gx, gy, gz], 1).cpu().numpy(), gp, rtol=1e-12, atol=1e-9 * np.abs(gp).max())
    assert float(buf[:shift].abs().sum()) == 0 and float(buf[shift + total:].abs().sum()) == 0
