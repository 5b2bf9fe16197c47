"""The tiled Barnes-Hut expansion against an FP64 walk of the same tree
(oracle restatement) where it can go wrong: target counts about a warp and
about the switch between one and four warps per 32 targets, halos sharing a
warp, everything opened (the node stack runs full), leaves longer than a
tile, coincident particles, and squared distances below the normal floats.

Tolerance: all terms have one sign, so the relative error of the sum is at
most that of a term: rsqrt 2^-22.9, the squared distance's 2^-22 halved, and
five roundings, together below 6e-7; the Kahan sums and the final rounding
add 2^-23.  The bar is 1e-6, as for the batched potential."""
import numpy as np
import pytest
import torch

from galaxyfinder_b200 import batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda_device):
    c = batch.Context(0)
    yield c
    c.close()


def _check(ctx, restatement, counts, p, m, theta2, ndirect=0, sample=400, seed=0):
    ps = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    pos4 = np.concatenate([p, m[:, None]], 1).astype(np.float32)
    t = batch.tree_build_export(ctx, ps, pos4, theta2=theta2)
    _, raw = batch.self_potential(ctx, ps, pos4, theta2=theta2, ndirect=ndirect)
    raw = raw.cpu().numpy().astype(np.float64)
    n = len(p)
    sel = np.sort(np.random.default_rng(seed).choice(n, min(n, sample), replace=False))
    h = np.searchsorted(ps, sel, "right") - 1
    op = (np.asarray(counts)[h] < ndirect).astype(np.int32)
    want = restatement.tree_potential(t["bh"], t["pos"], pos4[sel, :3], t["root"][h], t["rend"][h], op)
    zero = want == 0.0  # a halo of one particle, summed directly
    assert np.all(raw[sel][zero] == 0.0)
    fin = np.isfinite(want)  # (a lone particle's cell is singular in the reference too)
    assert np.array_equal(fin, np.isfinite(raw[sel]))
    ok = fin & ~zero
    err = np.abs(raw[sel] - want)[ok] / np.abs(want)[ok]
    assert err.size == 0 or err.max() < 1e-6, err.max()


def _cloud(rng, n):
    r = rng.random(n) ** 2 * 0.4
    v = rng.standard_normal((n, 3))
    return 0.5 + v / np.linalg.norm(v, axis=1, keepdims=True) * r[:, None]


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 64, 1000, 66303, 66336, 66400, 140001])
def test_target_counts(ctx, restatement, n):
    rng = np.random.default_rng(n)
    _check(ctx, restatement, [n], _cloud(rng, n), 10 ** rng.uniform(6, 8, n), 0.5, seed=n)


@pytest.mark.parametrize("ndirect", [0, 100])
def test_halos_sharing_a_warp(ctx, restatement, ndirect):
    rng = np.random.default_rng(7)
    counts = [5, 1, 40, 3, 130, 17, 99, 100, 101, 2, 700]
    n = sum(counts)
    _check(ctx, restatement, counts, _cloud(rng, n), 10 ** rng.uniform(6, 8, n), 0.5, ndirect, sample=n)


@pytest.mark.parametrize("n,theta2", [(3000, 1e-9), (150000, 1e-9), (20000, 0.02), (90000, 4.0)])
def test_opening_extremes(ctx, restatement, n, theta2):
    rng = np.random.default_rng(n)
    _check(ctx, restatement, [n], _cloud(rng, n), np.ones(n), theta2, sample=150)


@pytest.mark.parametrize("ncopy", [9, 10, 33, 1000])
def test_coincident_particles(ctx, restatement, ncopy):
    """ncopy particles at one place within a cloud: a leaf longer than a tile,
    pairs at zero distance left out.  The copies themselves are excluded: a
    node holding only copies has its centre on them, and the cell term there
    is singular in the reference too."""
    rng = np.random.default_rng(ncopy)
    p = _cloud(rng, 3000)
    p[:ncopy] = p[0]
    m = rng.random(3000) + 0.5
    ps = np.array([0, 3000])
    pos4 = np.concatenate([p, m[:, None]], 1).astype(np.float32)
    t = batch.tree_build_export(ctx, ps, pos4)
    _, raw = batch.self_potential(ctx, ps, pos4)
    sel = np.arange(ncopy, 3000)
    want = restatement.tree_potential(t["bh"], t["pos"], pos4[sel, :3], np.zeros(len(sel), np.int32),
                                      np.full(len(sel), t["rend"][0], np.int32))
    err = np.abs(raw.cpu().numpy()[sel] - want) / np.abs(want)
    assert err.max() < 1e-6, err.max()


@pytest.mark.parametrize("gap", [1e-16, 3e-20, 1e-23])
def test_tiny_separations(ctx, restatement, gap):
    """Pairs whose squared distance is a normal, a subnormal and a zero float
    (at 1e-23 the FP32 square underflows and the pair is left out, as by the
    float test r^2 > 0 of the reference's particle term)."""
    rng = np.random.default_rng(3)
    p = _cloud(rng, 500)
    p[0] = 0.0
    p[1] = [gap, 0.0, 0.0]
    pos4 = np.concatenate([p, np.ones((500, 1))], 1).astype(np.float32)
    q = pos4.astype(np.float64)
    _, raw = batch.self_potential(ctx, [0, 500], pos4, ndirect=1000)
    d = np.linalg.norm(q[:2, None, :3] - q[None, :, :3], axis=-1)
    with np.errstate(divide="ignore"):
        w = np.where(d > (1e-21 if gap == 1e-23 else 0), 1.0 / d, 0.0)
    want = -w.sum(1)
    got = raw.cpu().numpy()[:2]
    # a subnormal square has 23 - log2(2^-126 / r2) significant bits left
    bits = 1e-6 if gap > 1e-19 else 0.5 * 2.0 ** -149 / gap ** 2 + 1e-6
    assert np.all(np.abs(got - want) <= bits * np.abs(want))


def test_external_targets_in_any_order(ctx, restatement):
    """The potential of one set at scattered points (External_Halo_Potent:
    direct sum below 1000 targets, the tree above) against FP64 walks of the
    same sources' tree."""
    from galaxyfinder_b200 import dropin
    rng = np.random.default_rng(9)
    src, m = _cloud(rng, 5000), np.ones(5000, np.float32)
    t = batch.tree_build_export(ctx, [0, 5000], np.concatenate([src, m[:, None]], 1).astype(np.float32))
    ph, bg = dropin.physics(), dropin.bg_potent(5000.0)
    for nt in (999, 1000):
        r = rng.random((nt, 3))
        pe = dropin.External_Halo_Potent(r, np.ones(nt, np.float32), src, m)
        phi = restatement.tree_potential(t["bh"], t["pos"], r.astype(np.float32), np.zeros(nt, np.int32),
                                         np.full(nt, t["rend"][0], np.int32), np.full(nt, int(nt < 1000), np.int32))
        assert np.abs(pe / (phi * ph["potentfact"] + bg) - 1).max() < 1e-6
