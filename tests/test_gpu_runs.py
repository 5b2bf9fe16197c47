"""Extents, mesh boxes and the tiled deposit where a warp's run or a block's
chunk of consecutive particles meets halo boundaries: frames against numpy
exactly, and the density at the particles against the same stage with the
meshes kept on chip, which uses neither boxes nor tiles."""
import numpy as np
import pytest
import torch

from galaxyfinder_b200 import _lib, batch

pytestmark = pytest.mark.gpu

BATCHES = {
    "small": list(range(1, 70)),
    "edges": [31, 32, 33, 0, 0, 95, 96, 97, 127, 128, 129, 1, 255, 256, 257, 0],
    "steps": [32767, 1, 32768, 700],          # around a second step per warp
    "runs": [131072, 60, 131, 140000],        # four steps per warp, several chunks of the deposit
    "chunks": [400000, 3, 300001],            # chunks of more than a particle per thread
}


def _halos(counts, seed=3):
    rng = np.random.default_rng(seed)
    parts = []
    for c in counts:
        v = rng.standard_normal((c, 3))
        r = rng.random(c) ** 2 * 0.3
        p = 50 + 49 * (2 * rng.random(3) - 1) + v / np.maximum(np.linalg.norm(v, axis=1, keepdims=True), 1e-9) * r[:, None]
        parts.append(np.mod(p, 100.0))
    return parts


@pytest.mark.parametrize("name", BATCHES)
def test_runs_and_chunks(cuda_device, name):
    parts = _halos(BATCHES[name])
    ps = np.concatenate([[0], np.cumsum([len(p) for p in parts])]).astype(np.int64)
    xyz, n = np.concatenate(parts), int(ps[-1])
    dev = cuda_device
    t = lambda a, d: torch.from_numpy(np.ascontiguousarray(a)).to(dev, d)  # noqa: E731
    mass = 1 + np.random.default_rng(4).random(n)
    db = batch.DeviceBatch(*(t(xyz[:, a], torch.float64) for a in range(3)), t(mass, torch.float64),
                           torch.full((n,), _lib.TYPE_DM, dtype=torch.int32, device=dev), t(ps, torch.int64))
    ctx = batch.Context(0)
    outs = []
    for onchip in (False, True):
        cfg = batch.stage_config(mesh=batch.mesh_rule(mode=_lib.MESH_FIXED, nfixed=64, rg=2.0, rg_in_cells=True),
                                 mesh_onchip=onchip)
        out = batch.StageBuffers(n, 32, dev, keep_positions=True)
        torch.cuda.synchronize()
        batch.stage_run(ctx, db, cfg, out)
        outs.append(out)
    ctx.close()
    got = np.stack([outs[0].xr.cpu().numpy(), outs[0].yr.cpu().numpy(), outs[0].zr.cpu().numpy()], 1)
    for h, p in enumerate(parts):
        if not len(p):
            continue
        q = p.copy()
        for a in range(3):  # Dump2BP: unwrapped where the halo straddles the box
            s = np.where(q[:, a] < 50.0, q[:, a] + 100.0, q[:, a])
            if q[:, a].max() - q[:, a].min() > 50.0:
                q[:, a] = s
        np.testing.assert_array_equal(got[ps[h]:ps[h + 1]], q - q.min(0))
    # float sums of up to 400,000 terms per cell in two orders: sqrt(t) u of
    # the largest cell, which the smoothing averages
    a, b = (o.dens_mesh.cpu().numpy() for o in outs)
    for h in range(len(parts)):
        s = slice(ps[h], ps[h + 1])
        if len(a[s]):
            assert np.abs(a[s] - b[s]).max() <= 4e-5 * np.abs(b[s]).max(), h
