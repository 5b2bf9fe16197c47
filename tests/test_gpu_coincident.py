"""The potential of particles that share a place with enough others to fill a
node: finite, and the sum over the other particles, whatever way the node's
centre of mass rounds (in small halos, large ones and among other particles)."""
import numpy as np
import pytest
import torch

from galaxyfinder_b200 import batch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("core", [10, 16, 127, 128, 255, 257, 510, 5000])
@pytest.mark.parametrize("rest", [0, 7, 128, 3000])
@pytest.mark.parametrize("masses", ["equal", "any"])
def test_finite_and_equal_to_the_direct_sum(cuda_device, core, rest, masses):
    """theta^2 = 1e-6: every cell with an extent is opened by targets within
    1000 times its size, so the tree's error is below 1e-5 of the potential;
    particles at distance zero are left out, as in the reference's terms."""
    rng = np.random.default_rng(core + rest)
    p = np.concatenate([np.tile(rng.random(3), (core, 1)), rng.random((rest, 3))]).astype(np.float32)
    m = np.ones(len(p), np.float32) if masses == "equal" else (10 ** rng.uniform(-1, 1, len(p))).astype(np.float32)
    order = rng.permutation(len(p))
    p, m = p[order], m[order]
    ctx = batch.Context(0)
    _, raw = batch.self_potential(ctx, [0, len(p)], np.concatenate([p, m[:, None]], 1), theta2=1e-6)
    _, wide = batch.self_potential(ctx, [0, len(p)], np.concatenate([p, m[:, None]], 1), theta2=0.5)
    raw, wide = raw.cpu().numpy(), wide.cpu().numpy()
    ctx.close()
    x = torch.as_tensor(p, dtype=torch.float64, device=cuda_device)
    d2 = ((x[:, None] - x[None]) ** 2).sum(-1)
    want = -(torch.where(d2 > 0, d2, torch.inf).rsqrt() @ torch.as_tensor(m, dtype=torch.float64, device=cuda_device))
    want = want.cpu().numpy()
    assert np.isfinite(raw).all() and np.isfinite(wide).all()
    assert np.abs(raw - want).max() <= 1e-5 * np.abs(want).max()
    if rest == 0:
        assert (raw == 0).all() and (wide == 0).all()


@pytest.mark.parametrize("sizes", [(1, 1, 1), (1, 40, 1), (300, 1, 20)])
def test_lone_particles(cuda_device, sizes):
    """A halo of one particle has no potential of its own."""
    rng = np.random.default_rng(3)
    n = sum(sizes)
    q = np.concatenate([rng.random((n, 3)), np.ones((n, 1))], 1).astype(np.float32)
    ps = np.concatenate([[0], np.cumsum(sizes)])
    ctx = batch.Context(0)
    _, raw = batch.self_potential(ctx, ps, q)
    raw = raw.cpu().numpy()
    ctx.close()
    assert np.isfinite(raw).all()
    for h, s in enumerate(sizes):
        if s == 1:
            assert raw[ps[h]] == 0
