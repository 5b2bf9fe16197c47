"""Direct-convolution taps made on the host (few short axes) and on the device
(from 1024 terms on): meshes on both sides of the line against the FP64 spectral
smoothing, and no kernel for the taps of the smallest.

The bar of the sums: n products and additions of floats, n u of the largest value
per axis (u = 2^-24, taps of sum 1), and the taps' own rounding, u each."""
import json

import numpy as np
import pytest
import torch

from galaxyfinder_b200 import _lib, batch
from oracle import adjoint as oadj

pytestmark = pytest.mark.gpu


def _smooth(ctx, dims, a):
    d = np.zeros(1, _lib.MESH_DTYPE)
    d["nx"], d["ny"], d["nz"], d["ptype"], d["cellsize"], d["rg"] = *dims, 5, 0.004, 0.007
    den = torch.from_numpy(a.ravel()).to("cuda:0")
    _lib.check(_lib.lib().gf_gaussian_smooth(ctx.handle, 1, _lib.ptr(d),
                                             _lib.ptr(torch.from_numpy(d.view(np.uint8)).to("cuda:0")), _lib.ptr(den)))
    torch.cuda.synchronize()
    return den.cpu().numpy().reshape(a.shape)


@pytest.mark.parametrize("dims", [(1, 1, 1), (2, 3, 5), (7, 1, 9), (31, 7, 3), (32, 31, 7), (33, 3, 2), (18, 18, 18),
                                  (18, 19, 20), (30, 9, 7), (64, 31, 5), (128, 33, 31)])
def test_taps_of_short_axes(cuda_device, dims):
    nx, ny, nz = dims
    ctx = batch.Context(0)
    mesh = oadj.Mesh(nx, ny, nz, 0, 0, 0, 0.004, 0.007)
    a = np.zeros((nz, ny, mesh.mx), np.float32)
    a[:, :, :nx] = np.random.default_rng(nx).random((nz, ny, nx)) ** 4
    want = oadj.smooth(a.astype(np.float64), mesh)
    got = _smooth(ctx, dims, a)
    ctx.close()
    bar = sum((n + 1 if n not in (64, 128) else 14 * np.log2(n) * np.sqrt(2 * n)) for n in dims) * 2.0 ** -24
    assert np.abs(got - want)[:, :, :nx].max() <= bar * a.max()


def test_no_kernel_for_few_taps(cuda_device, tmp_path):
    ctx = batch.Context(0)
    names = {}
    for n in (20, 40):
        a = np.ones((n, n, 2 * (n // 2 + 1)), np.float32)
        acts = [torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA]
        with torch.profiler.profile(activities=acts) as prof:
            _smooth(ctx, (n, n, n), a)
        f = tmp_path / f"{n}.json"
        prof.export_chrome_trace(str(f))
        names[n] = [e["name"] for e in json.loads(f.read_text())["traceEvents"] if e.get("cat") == "kernel"]
    ctx.close()
    assert any("smooth_direct" in k for k in names[20])
    assert not any("axis_taps" in k for k in names[20]) and any("axis_taps" in k for k in names[40])
