"""The work that users have this framework do, as cases of one call each.

Every case goes through a public entry point (``galaxyfinder_b200.batch``,
``.autograd``, ``.dropin``) on seeded synthetic halos with the statistics of
``galaxyfinder_b200.synth``: NFW haloes with subhaloes and 20 % stars, counts
from N^-1.9, 5 % of the haloes across the periodic box, or Gaussian mixtures.
``prepare`` makes the inputs and the handles a program keeps (context, output
buffers, mesh plan, captured pipeline), ``run`` is one call, ``exact`` the same
outputs in 64 bits by plain torch where that takes seconds."""
from __future__ import annotations

import math

import numpy as np
import torch

from galaxyfinder_b200 import _lib, autograd, batch, dropin, synth

BOX = 100.0
RHO_C = 2.7755e11
DM_MASS = 1.0e8
STAR, DM = 1, 2
DEV = "cuda:0"


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the stage for one FoF group of the smallest kind a finder keeps: a
        # call that is all launches and waits
        dict(name="stage_group_120", kind="stage", nhalo=1, nmin=120, nmax=120, mesh="pow2", k=32),
        # one massive halo with the mesh fixed at 128^3, the single-halo
        # workload of the benchmark
        dict(name="stage_halo_131072", kind="stage", nhalo=1, nmin=131072, nmax=131072, mesh="fixed128", k=32),
        # a ragged batch as a rank of a shared catalogue gets: many small
        # halos, one that is large
        dict(name="stage_catalogue_256", kind="stage", nhalo=256, nmin=100, nmax=200_000, mesh="pow2", k=32),
        # the whole benchmark catalogue in one call, the throughput workload
        dict(name="stage_catalogue_4096", kind="stage", nhalo=4096, nmin=100, nmax=2_000_000, mesh="pow2", k=32),
        # the production loop: pinned host inputs in, all outputs back, the
        # chunks' captured stages overlapped
        dict(name="pipeline_e2e_1024", kind="pipeline", nhalo=1024, nmin=100, nmax=500_000, chunks=6),
        # stellar meshes at the reference's own rule (0.004 cMpc/h cells, any
        # length per axis), whole meshes kept: the input of peak finding
        dict(name="mesh_reference_48", kind="mesh", nhalo=48, nmin=300, nmax=60_000),
        # neighbour lists and densities alone, clumpy halo without a profile
        dict(name="knn_mixture_1m", kind="knn", n=1_000_003, clumps=64, k=32),
        # potential alone at the narrower opening angle, for the energy cuts
        dict(name="potential_cluster_300k", kind="potential", n=300_007, theta2=0.25),
        # differentiable mesh density: forward and backward, 256^3 mesh
        dict(name="grad_mesh_2m", kind="grad_mesh", n=2_000_000, clumps=64, mesh=256),
        # differentiable kNN density at probes: forward and backward
        dict(name="grad_probes_1m", kind="grad_probes", n=1_000_000, clumps=64, probes=4096),
        # the reference's own signatures on host arrays, one halo, as a
        # program linked with the library calls them
        dict(name="dropin_halo_36k", kind="dropin", n=36_001),
        # a captured stage replayed on a small batch that stays on the device,
        # as a time series of the same groups is run
        dict(name="graph_catalogue_64", kind="graph", nhalo=64, nmin=100, nmax=50_000),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["stage", "stage", "stage", "pipeline", "mesh", "knn", "potential", "grad_mesh", "grad_probes",
                       "dropin", "graph"])
    if kind == "stage":
        if rng.random() < 0.35:  # one halo of any size
            n = log(100, 1_500_000)
            return dict(kind=kind, nhalo=1, nmin=n, nmax=n, mesh="fixed128" if n > 5000 and rng.random() < 0.5 else "pow2",
                        k=rng.choice([32, 32, 20, 13]))
        return dict(kind=kind, nhalo=log(2, 3000), nmin=log(50, 200), nmax=log(5_000, 1_500_000), mesh="pow2",
                    k=rng.choice([32, 32, 20, 13]))
    if kind == "pipeline":
        return dict(kind=kind, nhalo=log(100, 2000), nmin=100, nmax=log(50_000, 500_000), chunks=rng.choice([3, 6, 12]))
    if kind == "mesh":
        return dict(kind=kind, nhalo=log(1, 48), nmin=300, nmax=log(3_000, 60_000))
    if kind == "knn":
        return dict(kind=kind, n=log(500, 1_500_000), clumps=log(1, 64), k=rng.choice([32, 20, 7]))
    if kind == "potential":
        return dict(kind=kind, n=log(500, 600_000), theta2=rng.choice([0.5, 0.25]))
    if kind == "grad_mesh":
        return dict(kind=kind, n=log(10_000, 2_000_000), clumps=log(4, 64), mesh=rng.choice([64, 128, 256]))
    if kind == "grad_probes":
        return dict(kind=kind, n=log(5_000, 1_000_000), clumps=log(4, 64), probes=log(256, 4096))
    if kind == "dropin":
        return dict(kind=kind, n=log(2_000, 60_000))
    return dict(kind=kind, nhalo=log(1, 400), nmin=100, nmax=log(2_000, 200_000))


# ------------------------------------------------------------------ the inputs
def _counts(case):
    """Particle counts of dN/dN_p ~ N_p^-1.9 at the middles of nhalo equal
    probabilities, in an order of no meaning, so that a case has the same
    shapes for every seed."""
    nhalo, nmin, nmax = case["nhalo"], case["nmin"], case["nmax"]
    a, rng = -0.9, np.random.default_rng(nhalo)
    u = (np.arange(nhalo) + 0.5) / nhalo
    c = np.floor((nmin ** a + u * (float(nmax) ** a - nmin ** a)) ** (1.0 / a) + 1e-6).astype(np.int64)
    return rng.permutation(np.clip(c, nmin, nmax))


def _r200(m):
    return (3.0 * np.asarray(m) / (4.0 * np.pi * 200.0 * RHO_C)) ** (1.0 / 3.0)


def _nfw(centre, r200, conc, counts, g):
    """Particles of NFW components: positions of sum(counts) particles, by
    bisection of the enclosed-mass profile."""
    rep = torch.as_tensor(counts, device=DEV)
    n = int(rep.sum())
    c = torch.repeat_interleave(torch.as_tensor(conc, device=DEV), rep)
    rv = torch.repeat_interleave(torch.as_tensor(r200, device=DEV), rep)
    ctr = torch.repeat_interleave(torch.as_tensor(centre, device=DEV), rep, dim=0)
    mu = lambda x: torch.log1p(x) - x / (1.0 + x)  # noqa: E731
    want = torch.rand(n, generator=g, device=DEV, dtype=torch.float64) * mu(c)
    lo, hi = torch.zeros_like(want), torch.ones_like(want)
    for _ in range(34):
        mid = 0.5 * (lo + hi)
        low = mu(c * mid) < want
        lo, hi = torch.where(low, mid, lo), torch.where(low, hi, mid)
    v = torch.randn((n, 3), generator=g, device=DEV, dtype=torch.float64)
    v /= v.norm(dim=1, keepdim=True)
    return ctr + (rv * 0.5 * (lo + hi))[:, None] * v


def _halos(counts, seed):
    """(x, y, z, mass, type, pstart) of NFW halos with subhalos and stars, as
    synth.catalogue makes them, on the GPU."""
    rng = np.random.default_rng(seed)
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + 17)
    counts = np.asarray(counts, np.int64)
    nh = len(counts)
    nstar = np.round(0.2 * counts).astype(np.int64)
    ndm = counts - nstar
    mtot = ndm * DM_MASS + nstar * 10 ** rng.uniform(6, 7, nh)
    r200 = _r200(mtot)
    conc = 10 ** (np.log10(6.0) + 0.15 * rng.standard_normal(nh))
    centre = rng.random((nh, 3)) * BOX
    wrap = np.flatnonzero(rng.random(nh) < 0.05)
    centre[wrap, rng.integers(0, 3, len(wrap))] = rng.uniform(-0.3, 0.3, len(wrap)) * r200[wrap]
    own, sub_c, sub_r, sub_k, sub_n = [], [], [], [], []
    host = ndm.copy()
    for h in np.flatnonzero(mtot > 5e10):
        ns = rng.poisson(mtot[h] / 1e11)
        a = -0.9
        f = 1e-5 * (1.0 + rng.random(ns) * (1e3 ** a - 1.0)) ** (1.0 / a)
        k = (f[np.cumsum(f) < 0.5] * ndm[h]).astype(np.int64)
        f, k = f[:len(k)][k > 0], k[k > 0]
        if not len(k):
            continue
        d = rng.standard_normal((len(k), 3))
        d *= (rng.uniform(0.1, 0.8, len(k)) * r200[h] / np.linalg.norm(d, axis=1))[:, None]
        own.append(np.full(len(k), h))
        sub_c.append(centre[h] + d)
        sub_r.append(r200[h] * f ** (1.0 / 3.0))
        sub_k.append(np.full(len(k), conc[h]))
        sub_n.append(k)
        host[h] -= int(k.sum())
    ids = np.arange(nh)
    comp = np.concatenate([ids, ids] + own)  # host halos, their stars, the subhalos
    pos = _nfw(np.concatenate([centre, centre] + sub_c), np.concatenate([r200, r200] + sub_r),
               np.concatenate([conc, 3.0 * conc] + sub_k), np.concatenate([host, nstar] + sub_n), g)
    cn = torch.as_tensor(np.concatenate([host, nstar] + sub_n), device=DEV)
    halo = torch.repeat_interleave(torch.as_tensor(comp, device=DEV), cn)
    kind = torch.repeat_interleave(torch.as_tensor((np.arange(len(comp)) // nh == 1).astype(np.int64), device=DEV), cn)
    order = torch.argsort(halo + torch.rand(len(halo), generator=g, device=DEV, dtype=torch.float64))
    pos, kind = torch.remainder(pos[order], BOX), kind[order]
    mstar = 10 ** (6.0 + torch.rand(len(kind), generator=g, device=DEV, dtype=torch.float64))
    mass = torch.where(kind == 1, mstar, torch.full_like(mstar, DM_MASS))
    typ = torch.where(kind == 1, STAR, DM).to(torch.int32)
    x, y, z = (pos[:, a].contiguous() for a in range(3))
    return x, y, z, mass, typ, np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)


def _mixture(n, clumps, seed):
    """Recentred FP64 positions (n, 3) of a Gaussian mixture (synth.config4):
    clumps of 5 to 50 kpc/h in a sphere of 0.5 Mpc/h."""
    rng = np.random.default_rng(seed)
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + 29)
    sig = np.exp(rng.uniform(np.log(0.005), np.log(0.05), clumps))
    w = np.exp(rng.uniform(0.0, np.log(100.0), clumps))
    cn = torch.as_tensor(rng.multinomial(n, w / w.sum()), device=DEV)
    d = rng.standard_normal((clumps, 3))
    ctr = d / np.linalg.norm(d, axis=1)[:, None] * (0.5 * rng.random(clumps) ** (1.0 / 3.0))[:, None]
    p = torch.repeat_interleave(torch.as_tensor(ctr, device=DEV), cn, dim=0)
    s = torch.repeat_interleave(torch.as_tensor(sig, device=DEV), cn)
    p = p + s[:, None] * torch.randn((n, 3), generator=g, device=DEV, dtype=torch.float64)
    p = p[torch.randperm(n, generator=g, device=DEV)]
    return p - p.min(0).values


def _one_halo(n, seed):
    """Recentred FP64 positions (n, 3), masses and types of one NFW halo."""
    x, y, z, m, t, _ = _halos([n], seed)
    p = _unwrapped(torch.stack([x, y, z], 1))
    return p - p.min(0).values, m, t


def _mesh_extent(case):
    """Extents that hold every halo of these counts, unlike along the axes."""
    return 2.06 * _r200(_counts(case) * DM_MASS)[:, None] * np.array([1.0, 1.03, 1.07])


def _rule(case):
    if case["mesh"] == "fixed128":
        return batch.mesh_rule(mode=_lib.MESH_FIXED, nfixed=128, rg=2.0, rg_in_cells=True)
    return batch.mesh_rule(mode=_lib.MESH_POW2, nmin=64, nmax=256, rg=2.0, rg_in_cells=True)


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("stage", "graph", "pipeline"):
        x, y, z, m, t, ps = _halos(_counts(case), seed)
    if kind == "stage":
        db = batch.DeviceBatch(x, y, z, m, t, torch.as_tensor(ps, device=DEV))
        return dict(kind=kind, ctx=batch.Context(0), db=db, cfg=batch.stage_config(mesh=_rule(case), knn_k=case["k"]),
                    out=batch.StageBuffers(db.n, case["k"], DEV))
    if kind == "graph":
        db, ctx = batch.DeviceBatch(x, y, z, m, t, torch.as_tensor(ps, device=DEV)), batch.Context(0)
        out = batch.StageBuffers(db.n, 32, DEV)
        return dict(kind=kind, out=out, graph=batch.StageGraph(ctx, db, batch.stage_config(mesh=_rule(dict(mesh="pow2"))), out))
    if kind == "pipeline":
        h = [a.cpu().numpy() for a in (x, y, z, m, t)]
        v = np.zeros(len(h[0]))  # the stage reads no velocities
        hb = synth.HaloBatch(x=h[0], y=h[1], z=h[2], vx=v, vy=v, vz=v, mass=h[3], type=h[4],
                             ids=np.arange(len(v)), pstart=ps)
        cfg = batch.stage_config(mesh=_rule(dict(mesh="pow2")), knn_k=32)
        return dict(kind=kind, pipe=batch.PipelinedStage(hb, cfg, nchunk=case["chunks"], graph=True))
    if kind == "mesh":
        x, y, z, m, t, ps = _halos(_counts(case), seed)
        p, _ = _recentred(x, y, z, ps)
        mesh, total = batch.plan_meshes(_mesh_extent(case), batch.mesh_rule(ptype=STAR))
        db = batch.DeviceBatch(*(p[:, a].contiguous() for a in range(3)), m, t, torch.as_tensor(ps, device=DEV))
        return dict(kind=kind, ctx=batch.Context(0), db=db, mesh=mesh, total=total)
    if kind == "knn":
        p = _mixture(case["n"], case["clumps"], seed)
        pos4 = torch.cat([p.float(), torch.ones((len(p), 1), device=DEV)], 1).contiguous()
        return dict(kind=kind, ctx=batch.Context(0), pos4=pos4, ps=np.array([0, len(p)], np.int64), k=case["k"])
    if kind == "potential":
        p, m, _ = _one_halo(case["n"], seed)
        pos4 = torch.cat([p.float(), m.float()[:, None]], 1).contiguous()
        return dict(kind=kind, ctx=batch.Context(0), pos4=pos4, ps=np.array([0, len(p)], np.int64), theta2=case["theta2"])
    if kind in ("grad_mesh", "grad_probes"):
        p = _mixture(case["n"], case["clumps"], seed)
        g = torch.Generator(device=DEV)
        g.manual_seed(int(seed) + 5)
        ctx, ps = batch.Context(0), np.array([0, len(p)], np.int64)
        x, y, z = (p[:, a].contiguous().requires_grad_() for a in range(3))
        s = dict(kind=kind, ctx=ctx, xyz=(x, y, z), ps=ps)
        if kind == "grad_mesh":
            rule = batch.mesh_rule(mode=_lib.MESH_FIXED, nfixed=case["mesh"], rg=1.5, rg_in_cells=True)
            mesh, total = batch.plan_meshes(p.max(0).values.cpu().numpy()[None], rule)
            m = torch.full((len(p),), DM_MASS, dtype=torch.float64, device=DEV).requires_grad_()
            up = torch.rand(len(p), generator=g, device=DEV)  # dL/drho
            return dict(s, m=m, plan=autograd.MeshPlan(ctx, ps, mesh, total), up=up)
        q = torch.randperm(len(p), generator=g, device=DEV)[:min(case["probes"], len(p))]
        return dict(s, q=q, up=torch.rand(len(q), generator=g, device=DEV))
    if kind == "dropin":
        p, m, t = (a.cpu().numpy() for a in _one_halo(case["n"], seed))
        bp = np.zeros(len(p), _lib.BP_DTYPE)
        bp["x"], bp["y"], bp["z"] = p.T
        bp["mass"], bp["type"] = m, t
        mesh, _ = batch.plan_meshes(p.max(0)[None], _rule(dict(mesh="pow2")))
        mm = mesh[0]
        den = np.zeros(dropin.mesh_floats(int(mm["nx"]), int(mm["ny"]), int(mm["nz"])), np.float32)
        return dict(kind=kind, bp=bp, p=p, m=m.astype(np.float32), mesh=mm, den=den)
    raise ValueError(kind)


# ------------------------------------------------------------------ the calls
def run(s):
    kind = s["kind"]
    if kind in ("stage", "graph"):
        if kind == "graph":
            s["graph"].run()
            o = s["out"]
        else:
            o = batch.stage_run(s["ctx"], s["db"], s["cfg"], s["out"])
        return dict(near=o.nearindex, dens_sph=o.dens_sph, dens_mesh=o.dens_mesh, penergy=o.penergy)
    if kind == "pipeline":
        _, end = s["pipe"].run_e2e()
        end.synchronize()
        s["pipe"].check()
        return [c["hout"] for c in s["pipe"].chunks]
    if kind == "mesh":
        den, rho = batch.mesh_stage(s["ctx"], s["db"], s["mesh"], s["total"])
        return dict(den=_cells(den, s["mesh"]), rho=rho)
    if kind == "knn":
        near, dens = batch.knn_density(s["ctx"], s["ps"], s["pos4"], s["k"])
        return dict(near=near, dens=dens)
    if kind == "potential":
        pe, raw = batch.self_potential(s["ctx"], s["ps"], s["pos4"], theta2=s["theta2"], ndirect=100)
        return dict(penergy=pe, raw=raw)
    if kind in ("grad_mesh", "grad_probes"):
        x, y, z = s["xyz"]
        if kind == "grad_mesh":
            rho = autograd.MeshDensityAt.apply(x, y, z, s["m"], s["plan"])
            return [rho.detach(), *torch.autograd.grad(rho, (x, y, z, s["m"]), s["up"])]
        rho = autograd.KnnDensity.apply(x, y, z, s["q"], 32, s["ctx"], s["ps"])
        return [rho.detach(), *torch.autograd.grad(rho, (x, y, z), s["up"])]
    mm, den = s["mesh"], s["den"]
    n3 = (int(mm["nx"]), int(mm["ny"]), int(mm["nz"]))
    o, cell = float(mm["xmin"]), float(mm["cellsize"])
    near, dens = dropin.findsphdensity(s["bp"], 32)
    den[:] = 0
    dropin.assign_density_TSC(s["bp"], *n3, o, o, o, cell, _lib.TYPE_ALL, den=den)
    dropin.gaussian_Smoothing(den, *n3, cell, float(mm["rg"]))
    rho = dropin.findDen(s["bp"], den, *n3, o, o, o, cell)
    return dict(near=near, dens=dens, rho=rho, pe=dropin.Self_Halo_Potent(s["p"], s["m"]))


def _cells(den, mesh):
    """The meshes' own cells, as views: the two padding floats of a row and
    the alignment gaps between meshes hold nothing (up to 16 halos of them)."""
    step = max(1, len(mesh) // 16)
    out = []
    for d in mesh[::step][:16]:
        nx, ny, nz = int(d["nx"]), int(d["ny"]), int(d["nz"])
        mx = 2 * (nx // 2 + 1)
        out.append(den[int(d["off"]):int(d["off"]) + mx * ny * nz].view(nz, ny, mx)[:, :, :nx])
    return out


def work(case):
    """Bytes: inputs read once, outputs written once (meshes, where they are
    outputs).  Flops: 32 neighbours' distances and kernels, the 27-cell
    stencils, three FFT pairs over the mesh, and about 25 (theta2 = 0.5) or 60
    (0.25) cells and as many particles per target and log2 n, at 20 and 10."""
    kind = case["kind"]
    if kind in ("stage", "graph", "pipeline"):
        n = int(_counts(case).sum())
        k = case.get("k", 32)
        return dict(bytes=n * (36 + 4 * k + 12), flops=n * (40.0 * k + 27 * 8 + 25 * 30 * math.log2(n)))
    if kind == "mesh":
        c = _counts(case)
        cells = float(np.prod(_mesh_extent(case) / 0.004 + 10, axis=1).sum())
        return dict(bytes=40.0 * c.sum() + 4 * cells, flops=cells * 2 * 5 * 3 * 7)
    n = case["n"]
    if kind == "knn":
        return dict(bytes=n * (16.0 + 4 * case["k"] + 4), flops=n * 40.0 * case["k"])
    if kind == "potential":
        return dict(bytes=n * 24.0, flops=n * 30.0 * (60 if case["theta2"] < 0.4 else 25) * math.log2(n))
    if kind == "grad_mesh":
        # x, y, z, m, dL/drho in, rho and four gradients out
        return dict(bytes=n * (32.0 + 4 + 4 + 32), flops=n * 27 * 30.0 + case["mesh"] ** 3 * 3.0 * 2 * 5 * 3 * 8)
    if kind == "grad_probes":
        return dict(bytes=n * (24.0 + 24), flops=case["probes"] * 32 * 60.0)
    return dict(bytes=n * (88.0 + 24 + 4 + 8 * 32 + 12), flops=n * (40.0 * 32 + 27 * 8 + 25 * 30 * math.log2(n)))


# ------------------------------------------------------------------ 64 bits
def _unwrapped(p):
    """Positions of one halo in the more compact of its periodic images."""
    s = torch.where(p < 0.5 * BOX, p + BOX, p)
    w, ws = p.max(0).values - p.min(0).values, s.max(0).values - s.min(0).values
    return torch.where((w > 0.5 * BOX) & (ws < w), s, p)


def _recentred(x, y, z, ps):
    """Positions (n, 3) of every halo from its minimum, and the extents."""
    p = torch.stack([x, y, z], 1)
    out, ext = torch.empty_like(p), []
    for a, b in zip(ps[:-1], ps[1:]):
        q = _unwrapped(p[a:b])
        out[a:b] = q - q.min(0).values
        ext.append(out[a:b].max(0).values)
    return out, torch.stack(ext)


def _w4(r, h):
    q = r / h
    near = -0.2387324 * ((2.0 - q) * q * q - 1.333333) / h ** 3
    return torch.where(q < 1.0, near, torch.where(q < 2.0, 0.07957747 * ((2.0 - q) / h) ** 3, torch.zeros_like(q)))


def _pairs(p, m=None, k=None, targets=None):
    """All pairs of one halo, 64 bits: the W4 density over the k nearest (and
    those) and the sum of -m/r over the others."""
    q = p if targets is None else p[targets]
    rows = max(1, min(len(q), 100_000_000 // len(p)))
    dens, near, phi = [], [], []
    for a in range(0, len(q), rows):
        c = q[a:a + rows]
        d2 = (c[:, None, 0] - p[None, :, 0]) ** 2
        for ax in (1, 2):
            d2 += (c[:, None, ax] - p[None, :, ax]) ** 2
        if k:
            d, i = torch.topk(d2, min(k, len(p)), dim=1, largest=False)
            r = d.sqrt()
            dens.append(_w4(r, r[:, -1:] / 2).sum(1))
            near.append(i)
        if m is not None:
            phi.append(-(torch.where(d2 > 0, d2, torch.inf).rsqrt_() @ m))
    cat = lambda v: torch.cat(v) if v else None  # noqa: E731
    return cat(dens), cat(near), cat(phi)


def _stencil(p, mesh):
    """(flat cells, weights) of the 27 cells of every particle."""
    cell, org = float(mesh["cellsize"]), [float(mesh[f]) for f in ("xmin", "ymin", "zmin")]
    nx, ny, _ = (int(mesh[f]) for f in ("nx", "ny", "nz"))
    i, w = [], []
    for a in range(3):
        t = (p[:, a] - org[a]) / cell
        c = torch.round(t.detach())
        r = t - c
        i.append(c.long())
        w.append((0.5 * (0.5 - r) ** 2, 0.75 - r * r, 0.5 * (0.5 + r) ** 2))
    for dz in range(3):
        for dy in range(3):
            for dx in range(3):
                yield (((i[2] + dz - 1) * ny + i[1] + dy - 1) * nx + i[0] + dx - 1, w[0][dx] * w[1][dy] * w[2][dz])


def _mesh_density(p, m, mesh):
    """Deposit, Gaussian filter and interpolation in 64 bits: (mesh, rho)."""
    nx, ny, nz = (int(mesh[f]) for f in ("nx", "ny", "nz"))
    den = torch.zeros(nx * ny * nz, dtype=torch.float64, device=p.device)
    for c, w in _stencil(p, mesh):
        den = den.index_add(0, c, m * w) if den.requires_grad or w.requires_grad or m.requires_grad else den.index_add_(0, c, m * w)
    den = den.view(nz, ny, nx) * (0.001 / 0.004) ** 3
    rg = float(np.float32(float(np.float32(mesh["rg"])) / float(mesh["cellsize"])))  # held in a float, as the reference has it
    f = lambda n, fr: (fr(n, device=p.device, dtype=torch.float64)) ** 2  # noqa: E731
    arg = f(nz, torch.fft.fftfreq)[:, None, None] + f(ny, torch.fft.fftfreq)[:, None] + f(nx, torch.fft.rfftfreq)
    s = torch.fft.irfftn(torch.fft.rfftn(den) * torch.exp(-(math.pi * rg) ** 2 * arg), s=(nz, ny, nx))
    rho = 0.0
    flat = s.reshape(-1)
    for c, w in _stencil(p, mesh):
        rho = rho + flat[c] * w
    return s, rho


def _physics(mvir, potentfact):
    """NFW background potential of a halo's mass (omega_m 0.3, h 0.7, z 0)."""
    om, G = float(np.float32(0.3)), 6.672e-8
    c = 14.5 * (mvir / 1.3e13) ** -0.15
    gc = 1.0 / (math.log(1 + c) - c / (1 + c))
    vv = 18 * math.pi ** 2 + 82 * (om - 1) - 39 * (om - 1) ** 2
    rvir = (3 * mvir / (4 * math.pi * vv * RHO_C)) ** 0.3333333333333
    return G * mvir / rvir * potentfact * (1 - gc * math.log(1 + c))


def _potentfact():
    h0 = float(np.float32(70.0) / np.float32(100.0))
    return 6.672e-8 * (1.989e33 / h0) / (1.0 / h0 * 3.0857e24)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("stage", "graph"):
        c = _counts(case)
        if case["nhalo"] > 400 or (c.astype(float) ** 2).sum() > 8e10:
            return None
        x, y, z, m, _, ps = _halos(c, seed)
        p, ext = _recentred(x, y, z, ps)
        mesh, _ = batch.plan_meshes(ext.cpu().numpy(), _rule(dict(mesh=case.get("mesh", "pow2"))))
        out, pf = ([], [], []), _potentfact()
        for h, (a, b) in enumerate(zip(ps[:-1], ps[1:])):
            # the tree and the neighbour search are defined on the FP32 positions
            dens, _, phi = _pairs(p[a:b].float().double(), m[a:b].float().double(), case.get("k", 32))
            out[0].append(dens)
            out[1].append(_mesh_density(p[a:b], m[a:b], mesh[h])[1])
            out[2].append(phi * pf + _physics(float(m[a:b].sum()), pf))
        return dict(near=None, dens_sph=torch.cat(out[0]), dens_mesh=torch.cat(out[1]), penergy=torch.cat(out[2]))
    if kind == "mesh":
        s = prepare(case, seed)
        db, ps, den, rho = s["db"], s["db"].pstart.cpu().numpy(), [], []
        p = torch.stack([db.x, db.y, db.z], 1)
        step = max(1, len(s["mesh"]) // 16)
        for h, (a, b) in enumerate(zip(ps[:-1], ps[1:])):
            star = (db.type[a:b] == STAR).double()
            d, r = _mesh_density(p[a:b], db.mass[a:b] * star, s["mesh"][h])
            rho.append(r)
            if h % step == 0 and h // step < 16:
                den.append(d)
        return dict(den=den, rho=torch.cat(rho))
    if kind == "knn":
        if case["n"] > 250_000:
            return None
        s = prepare(case, seed)
        return dict(near=None, dens=_pairs(s["pos4"][:, :3].double(), None, case["k"])[0])
    if kind == "potential":
        if case["n"] > 350_000:
            return None
        s = prepare(case, seed)
        phi = _pairs(s["pos4"][:, :3].double(), s["pos4"][:, 3].double())[2]
        return dict(penergy=phi, raw=phi)
    if kind == "grad_mesh":
        s = prepare(case, seed)
        x, y, z = s["xyz"]
        rho = _mesh_density(torch.stack([x, y, z], 1), s["m"], s["plan"].mesh[0])[1]
        return [rho.detach(), *torch.autograd.grad(rho, (x, y, z, s["m"]), s["up"].double())]
    if kind == "grad_probes":
        s = prepare(case, seed)
        x, y, z = s["xyz"]
        p = torch.stack([x, y, z], 1)
        # lists and forward densities are those of the FP32 positions, the
        # gradient is taken at the FP64 ones
        dens, near, _ = _pairs(p.detach().float().double(), None, 32, s["q"])
        r2 = ((p[s["q"]][:, None] - p[near]) ** 2).sum(-1)
        own = near == s["q"][:, None]
        r = torch.where(own, torch.zeros_like(r2), torch.where(own, torch.ones_like(r2), r2).sqrt())
        rho = _w4(r, r[:, -1:] / 2).sum(1)
        return [dens, *torch.autograd.grad(rho, (x, y, z), s["up"].double())]
    if kind == "dropin":
        s = prepare(case, seed)
        p = torch.as_tensor(s["p"], device=DEV)
        m = torch.as_tensor(s["m"], device=DEV).double()
        dens, _, phi = _pairs(p.float().double(), m, 32)
        rho = _mesh_density(p, torch.as_tensor(np.ascontiguousarray(s["bp"]["mass"]), device=DEV), s["mesh"])[1]
        pf = _potentfact()
        return dict(near=None, dens=dens, rho=rho, pe=phi * pf + _physics(float(m.sum()), pf))
    return None  # the pipeline runs the stage's kernels
