"""Faint pencils beside bright ones: the register transforms filter two real
pencils as one complex pencil, and the rounding errors of either half are as
large as the brighter half's.  A pair is two neighbouring pencils, so a faint
value is off by the errors of its own pencil and its neighbour's, at any
distance from a bright one beyond that.

The bars bound the FFT's rounding: forward and back, a pencil pair x of n cells
is off by at most 2 log2(n) (4 + sqrt(2) + 1) u |x|_2 < 14 u log2(n) |x|_2
(Higham, Accuracy and Stability of Numerical Algorithms, theorem 24.2), u =
2^-24."""
import numpy as np
import pytest
import torch

from galaxyfinder_b200 import _lib, autograd, batch
from oracle import adjoint as oadj

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


@pytest.fixture(scope="module")
def ctx(cuda_device):
    c = batch.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("n", [64, 128, 256])
@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("bright", [0, 5, 16, 38, 69])
@pytest.mark.parametrize("shift", [0, 1], ids=["aligned", "odd"])
def test_faint_pencils(ctx, n, axis, bright, shift):
    """70 pencils along one axis, one of them 1e7 times the others, through a
    filter of radius zero (the identity); the mesh at an 8-byte boundary and
    between two."""
    dims = [70 if axis == 2 else 1] * 3
    dims[0 if axis else 1] = 70
    dims[axis] = n
    if axis == 2:
        dims[1] = 1
    nx, ny, nz = dims
    rng = np.random.default_rng(n + bright)
    mx = 2 * (nx // 2 + 1)
    a = np.zeros((nz, ny, mx), np.float32)
    v = rng.uniform(0.5, 1.0, (nz, ny, nx))
    sel = [slice(None)] * 3  # [z, y, x]
    sel[1 if axis == 0 else 2] = bright
    v[tuple(sel)] *= 1e7
    a[:, :, :nx] = v
    d = np.zeros(1, _lib.MESH_DTYPE)
    d["nx"], d["ny"], d["nz"], d["ptype"], d["cellsize"], d["rg"] = nx, ny, nz, 5, 0.004, 0.0
    room = torch.zeros(a.size + 2, dtype=torch.float32, device="cuda:0")
    den = room[shift:shift + a.size]
    den.copy_(torch.from_numpy(a.ravel()))
    _lib.check(_lib.lib().gf_gaussian_smooth(ctx.handle, 1, _lib.ptr(d),
                                             _lib.ptr(torch.from_numpy(d.view(np.uint8)).to("cuda:0")), _lib.ptr(den)))
    torch.cuda.synchronize()
    got = den.cpu().numpy().reshape(a.shape)[:, :, :nx]
    err = np.abs(got.astype(np.float64) - a[:, :, :nx]).max(axis=(0, 2) if axis == 0 else (0, 1))
    faint = np.abs(np.arange(70) - bright) > 1
    assert err[faint].max() <= 14 * U * np.log2(n) * np.sqrt(2.0 * n)
    assert err.max() <= 14 * U * np.log2(n) * np.sqrt(2.0 * n) * 1e7


def _clump_and_isolated(n):
    """A clump of 1e7 times an isolated particle's mass on an n^3 mesh, and
    isolated particles in its z plane, 20 cells from it in y, every three
    cells in x but for those whose columns hold the clump's own tail (a
    filter of two cells: exp(-d^2/4) of the clump at d cells).  Positions in
    the halo's frame, masses, the isolated ones' indices, the mesh."""
    ext = 1.0
    rule = batch.mesh_rule(mode=_lib.MESH_FIXED, nfixed=n, rg=2.0, rg_in_cells=True)
    mesh, _ = batch.plan_meshes(np.full((1, 3), ext), rule)
    cell, o = float(mesh[0]["cellsize"]), float(mesh[0]["xmin"])
    lo, hi = int(np.ceil(-o / cell)) + 1, int(np.floor((ext - o) / cell)) - 1
    ic, jc, kc = n // 2, lo + 8, n // 2
    i = np.array([i for i in range(lo, hi) if i % 3 == 0 and abs(i - ic) >= 10])
    cells = np.concatenate([[[ic + 0.2, jc - 0.1, kc + 0.3]] * 64,
                            np.stack([i + 0.1, np.full(len(i), jc + 20.2), np.full(len(i), kc + 0.3)], 1)])
    p = np.concatenate([cells * cell + o, [[0.0] * 3, [ext] * 3]])
    m = np.concatenate([np.full(64, 1e7 / 64), np.ones(len(i) + 2)])
    return p, m, np.arange(64, 64 + len(i)), mesh[0], rule


@pytest.mark.parametrize("n", [64, 128, 256])
@pytest.mark.parametrize("graph", [False, True], ids=["stage", "replay"])
def test_isolated_particles_stage(ctx, n, graph):
    """The box passes.  A row through the isolated particles holds one in
    three cells (norm below sqrt(n / 3) of a value), their columns one."""
    p, m, iso, d, rule = _clump_and_isolated(n)
    mesh = oadj.Mesh.from_desc(d)
    want = oadj.find_den(p, oadj.smooth(oadj.tsc(p, m, mesh), mesh), mesh)[iso]
    db = batch.DeviceBatch.from_arrays(*(p.T + 20.0), m, np.full(len(p), 2), [0, len(p)])
    cfg = batch.stage_config(mesh=rule, do_potential=False)
    out = batch.StageBuffers(db.n, 32, db.x.device)
    if graph:
        g = batch.StageGraph(ctx, db, cfg, out)
        out.dens_mesh.zero_()
        g.run()
    else:
        batch.stage_run(ctx, db, cfg, out)
    torch.cuda.synchronize()
    rel = np.abs(out.dens_mesh.cpu().numpy()[iso] - want) / want
    if graph:
        g.close()
    assert rel.max() <= 14 * U * np.log2(n) * (np.sqrt(2 * n / 3.0) + 2 * 2.3)


@pytest.mark.parametrize("n", [64, 128, 256])
def test_isolated_particles_gradient(ctx, n):
    """The whole-mesh passes of MeshDensityAt, forward and backward: densities
    and mass gradients of the isolated particles, with the clump's weights
    1e7 times theirs in the loss."""
    p, m, iso, d, rule = _clump_and_isolated(n)
    mesh = oadj.Mesh.from_desc(d)
    S = oadj.smooth(oadj.tsc(p, m, mesh), mesh)
    want = oadj.find_den(p, S, mesh)[iso]
    up = np.ones(len(p))
    up[:64] = 1e7 / 64
    _, gS = oadj.find_den_grad(p, S, mesh, up)
    _, want_m = oadj.tsc_grad(p, m, mesh, oadj.smooth(gS, mesh))
    plan = autograd.MeshPlan(ctx, np.array([0, len(p)], np.int64), np.array([d]), _floats(mesh))
    t = [torch.tensor(a, dtype=torch.float64, device="cuda:0", requires_grad=True) for a in (*p.T, m)]
    rho = autograd.MeshDensityAt.apply(*t, plan)
    gm = torch.autograd.grad(rho, t[3], torch.tensor(up, dtype=torch.float32, device="cuda:0"))[0]
    bar = 14 * U * np.log2(n) * (np.sqrt(2 * n / 3.0) + 2 * 2.3)
    rel = np.abs(rho.detach().cpu().numpy()[iso] - want) / want
    rel_m = np.abs(gm.cpu().numpy()[iso] - want_m[iso]) / np.abs(want_m[iso])
    assert rel.max() <= bar and rel_m.max() <= bar


def _floats(mesh):
    return mesh.mx * mesh.ny * mesh.nz
