"""The octree build where its two parts meet: halos and nodes about the 256
particles below which one warp builds a subtree, batches that mix both sizes
and halos without particles, coincident particles and chains of nodes that
start with the same particle.  Every node of the exported tree is checked
against the node rule (nnost.c:105-197, ost.c:532-640) on its own particles."""
import numpy as np
import pytest

from galaxyfinder_b200 import batch
from galaxyfinder_b200._lib import GFError

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda_device):
    c = batch.Context(0)
    yield c
    c.close()


def _check(ctx, halos, theta2=0.5):
    counts = [len(h) for h in halos]
    ps = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    rng = np.random.default_rng(1)
    m = 10 ** rng.uniform(0, 1, ps[-1])
    pos4 = np.concatenate([np.concatenate(halos), m[:, None]], 1).astype(np.float32)
    t = batch.tree_build_export(ctx, ps, pos4, theta2=theta2)
    kn, bh, tp = t["knn"], t["bh"], t["pos"]
    np.testing.assert_array_equal(tp, pos4[t["perm"]])
    nodes = 0
    for h in range(len(halos)):
        a, b = ps[h], ps[h + 1]
        assert np.array_equal(np.sort(t["perm"][a:b]), np.arange(a, b))
        r, e = int(t["root"][h]), int(t["rend"][h])
        assert r == nodes and kn[r]["count"] == b - a and kn[r]["parent"] == -1 and e == kn[r]["skip"]
        nodes = e
        i = r
        for i in range(r, e):
            k = kn[i]
            s0, c = int(k["lstart"]), int(k["count"])
            if c == 0:
                assert i == r and e == r + 1
                continue
            P = tp[s0:s0 + c].astype(np.float64)
            mass = P[:, 3].sum()
            com = (P[:, :3] * P[:, 3:]).sum(0) / mass
            # sums of doubles in any order
            assert np.abs(bh[i]["com"] - com).max() < 1e-13 * max(1.0, np.abs(com).max())
            assert np.array_equal(k["lo"], tp[s0:s0 + c, :3].min(0)) and np.array_equal(k["hi"], tp[s0:s0 + c, :3].max(0))
            d = P[:, :3] - bh[i]["com"]
            r2 = (d * d).sum(1).max()
            # float offsets, squares and sums of the size, then a division
            assert abs(bh[i]["open_r2"] * theta2 - r2) <= 8 * 2.0 ** -24 * r2 + 1e-30
            q = np.stack([d[:, 0] ** 2, d[:, 1] ** 2, d[:, 2] ** 2, d[:, 0] * d[:, 1], d[:, 0] * d[:, 2],
                          d[:, 1] * d[:, 2]], 1)
            scale = (P[:, 3:] * np.abs(q)).sum(0)
            assert np.all(np.abs(bh[i]["q"] - (P[:, 3:] * q).sum(0)) <= (c + 8) * 2.0 ** -24 * scale + 1e-30)
            oct_ = (P[:, :3] > bh[i]["com"]) @ np.array([1, 2, 4])
            big = [o for o in range(8) if np.sqrt(r2) > 0.5e-6 and (oct_ == o).sum() >= 10]
            # [loose | children in octant order], consecutive in preorder
            at, j = s0 + int(k["lcount"]), i + 1
            assert not np.isin(oct_[:k["lcount"]], big).any()
            for o in big:
                n = int((oct_ == o).sum())
                assert kn[j]["lstart"] == at and kn[j]["count"] == n and kn[j]["parent"] == i
                assert np.all(oct_[at - s0:at - s0 + n] == o)
                at, j = at + n, int(kn[j]["skip"])
            assert at == s0 + c and j == k["skip"]
    assert nodes == t["nnode"]


def _cloud(rng, n):
    v = rng.standard_normal((n, 3))
    return 0.5 + v / np.linalg.norm(v, axis=1, keepdims=True) * (rng.random(n) ** 2 * 0.4)[:, None]


@pytest.mark.parametrize("n", [1, 2, 9, 10, 11, 32, 33, 255, 256, 257, 300, 1000, 2049, 8000, 40000])
def test_one_halo(ctx, n):
    _check(ctx, [_cloud(np.random.default_rng(n), n)])


def test_mixed_batch(ctx):
    rng = np.random.default_rng(2)
    counts = [0, 300, 0, 0, 5, 256, 257, 0, 10000, 1, 40, 3000, 255, 0]
    _check(ctx, [_cloud(rng, c) for c in counts])


@pytest.mark.parametrize("n", [200, 400, 5000])
def test_coincident_particles(ctx, n):
    rng = np.random.default_rng(n)
    p = _cloud(rng, n)
    p[: n // 2] = p[0]
    _check(ctx, [p, np.repeat(p[:1], n, 0), p[rng.permutation(n)]])


@pytest.mark.parametrize("n", [120, 600])
def test_chains(ctx, n):
    """Shells of geometrically shrinking radius about one corner: every level
    strips a few particles, so nodes nest deeply and start together."""
    rng = np.random.default_rng(n)
    r = 0.4 * 0.85 ** np.arange(n)
    _check(ctx, [0.5 + np.abs(rng.standard_normal((n, 3))) * r[:, None], 0.5 - r[:, None] * np.ones(3)])


@pytest.mark.parametrize("n", [200, 5000, 60000])
def test_extent_rounding(ctx, n):
    """max |x - com|^2 of every node to the bit, whichever kernel built it:
    fma(z, z, fma(x, x, y y)) of float offsets (a sum of a float and an exact
    product of two in doubles, rounded once more: equal but for ties within
    2^-29 of a unit, which the seeds do not hit)."""
    p = np.concatenate([_cloud(np.random.default_rng(n), n), np.ones((n, 1))], 1).astype(np.float32)
    t = batch.tree_build_export(ctx, np.array([0, n], np.int64), p, theta2=0.5)
    for k, b in zip(t["knn"], t["bh"]):
        P = t["pos"][k["lstart"]:k["lstart"] + k["count"], :3].astype(np.float64)
        d = (P - b["com"]).astype(np.float32)
        x, y, z = (d[:, a].astype(np.float64) for a in range(3))
        a = (x * x + (d[:, 1] * d[:, 1]).astype(np.float64)).astype(np.float32)
        r2 = (z * z + a.astype(np.float64)).astype(np.float32)
        assert b["open_r2"] == 2.0 * r2.max()


@pytest.mark.parametrize("n", [100, 300])
def test_endless_chain_is_refused(ctx, n):
    """One particle at infinity puts every centre of mass there: all particles
    fall into one octant on every level, and the build stops with an error."""
    p = _cloud(np.random.default_rng(n), n)
    p[n // 2] = np.inf
    with pytest.raises(GFError, match="deeper than"):
        _check(ctx, [p])


@pytest.mark.parametrize("n", [8191, 8192, 8193])
def test_numbering_of_small_batches(ctx, n):
    """Both sides of the batch size up to which one block numbers the nodes,
    with halos without particles at the ends and between."""
    rng = np.random.default_rng(n)
    _check(ctx, [_cloud(rng, c) for c in (0, 3000, 0, 0, 12, 700, n - 3712, 0)])
