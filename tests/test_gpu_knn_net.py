"""The sorted-list kNN kernel at the sizes where it can go wrong: the switches
between one, two and four lanes per query, lists shorter than 32, halos that
share a warp or are smaller than k, distances closer than a list key's step
(7.6e-6, 1.5e-5 with four lanes), many equal distances and many equal
positions.  Lists and densities are bit-exact by construction, so every
comparison with the exact oracle is for equality."""
import numpy as np
import pytest

from galaxyfinder_b200 import batch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(cuda_device):
    c = batch.Context(0)
    yield c
    c.close()


def _check(ctx, restatement, halos, k, method="grid"):
    ps = np.concatenate([[0], np.cumsum([len(p) for p in halos])]).astype(np.int64)
    pos4 = np.concatenate([np.concatenate([p, np.ones((len(p), 1), np.float32)], 1) for p in halos]).astype(np.float32)
    near, dens = batch.knn_density(ctx, ps, pos4, k)
    near, dens = near.cpu().numpy(), dens.cpu().numpy()
    for h, p in enumerate(halos):
        a, b = ps[h], ps[h + 1]
        kk = min(k, len(p))
        idx, d2 = restatement.knn(p[:, 0], p[:, 1], p[:, 2], kk, method)
        np.testing.assert_array_equal(near[a:b, :kk], idx, err_msg=f"halo {h}")
        assert np.all(near[a:b, kk:] == -1)
        np.testing.assert_array_equal(dens[a:b], restatement.sph_density(d2), err_msg=f"halo {h}")


def _cloud(rng, n):
    r = rng.random(n) ** 2 * 0.4
    v = rng.standard_normal((n, 3))
    return (0.5 + v / np.linalg.norm(v, axis=1, keepdims=True) * r[:, None]).astype(np.float32)


# 24 resident warps on 148 SMs: four lanes up to 28,416 particles, two up to 142,080
@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 31, 32, 33, 63, 127, 500, 28416, 28417, 142080, 142081])
def test_sizes(ctx, restatement, n):
    _check(ctx, restatement, [_cloud(np.random.default_rng(n), n)], 32)


@pytest.mark.parametrize("n", [40, 3000, 60000, 150000])
@pytest.mark.parametrize("k", [1, 2, 3, 5, 13, 20, 30, 31])
def test_short_lists(ctx, restatement, n, k):
    _check(ctx, restatement, [_cloud(np.random.default_rng(k), n)], k)


@pytest.mark.parametrize("scale", [1, 60])
@pytest.mark.parametrize("k", [32, 10])
def test_halos_sharing_a_warp(ctx, restatement, scale, k):
    rng = np.random.default_rng(11)
    counts = [5, 1, 40, 3, 33, 17, 31, 32, 2, 700, 9, 1200 * scale, 8, 1500 * scale, 6]
    _check(ctx, restatement, [_cloud(rng, c) for c in counts], k)


@pytest.mark.parametrize("n", [3000, 40000, 160000])
@pytest.mark.parametrize("eps", [1e-7, 3e-6, 1e-5])
def test_near_ties(ctx, restatement, n, eps):
    """Shells about random centres, 48 particles each at distances equal to
    within eps: the 32nd place lies among them."""
    rng = np.random.default_rng(n)
    m = n // 49
    c = _cloud(rng, m).astype(np.float64)
    v = rng.standard_normal((m, 48, 3))
    v /= np.linalg.norm(v, axis=-1, keepdims=True)
    p = c[:, None] + v * (1e-4 * (1 + eps * rng.random((m, 48, 1))))
    p = np.concatenate([c, p.reshape(-1, 3)]).astype(np.float32)
    _check(ctx, restatement, [p[rng.permutation(len(p))]], 32)


@pytest.mark.parametrize("side", [14, 34, 54])
def test_lattices(ctx, restatement, side):
    g = np.arange(side, dtype=np.float32) * np.float32(2.0 ** -7)
    p = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3)
    _check(ctx, restatement, [p[np.random.default_rng(side).permutation(len(p))]], 32)


@pytest.mark.parametrize("n,copies", [(2000, 40), (2000, 700), (40000, 100), (160000, 40)])
def test_equal_positions(ctx, restatement, n, copies):
    rng = np.random.default_rng(copies)
    p = _cloud(rng, n)
    p[: n // 2] = p[rng.integers(0, max(1, n // (2 * copies)), n // 2)]
    _check(ctx, restatement, [p[rng.permutation(n)]], 32, "brute" if n <= 2000 else "grid")


def test_probe_queries(ctx, restatement):
    """gf_knn_query spreads few queries over the warps and keeps 32 in a row
    where there are many."""
    from galaxyfinder_b200 import autograd
    import torch
    rng = np.random.default_rng(4)
    p = _cloud(rng, 400000)
    idx = None
    for nq in (1, 33, 4096, 300001):
        q = rng.permutation(len(p))[:nq]
        xyz = [torch.as_tensor(p[:, a].astype(np.float64), device="cuda:0") for a in range(3)]
        near, dens = autograd.knn_query(ctx, [0, len(p)], *xyz, q, 32)
        if idx is None:
            idx, d2 = restatement.knn(p[:, 0], p[:, 1], p[:, 2], 32)
            rho = restatement.sph_density(d2)
        np.testing.assert_array_equal(near.cpu().numpy(), idx[q])
        np.testing.assert_array_equal(dens.cpu().numpy(), rho[q])
