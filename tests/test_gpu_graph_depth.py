"""The planned depth of a captured stage where the deepest nodes hold more than
256 particles and have no child: a halo with many particles in one place, and
around it shells of five, each a hundredth of the one before, that go to no
child (a node's child needs 10 particles).  Every level of such a tree is one
node of more than 256."""
import numpy as np
import pytest
import torch

from galaxyfinder_b200 import _lib, batch, synth

pytestmark = pytest.mark.gpu

FIELDS = ("nearindex", "dens_sph", "dens_mesh", "penergy", "phi")


def _nested(core, shells, seed):
    """Positions (n, 3) from the core at the origin: shell k along the diagonal
    at 10^(-2 k)."""
    rng = np.random.default_rng(seed)
    out = [np.zeros((core, 3))]
    for k in range(shells):
        out.append(100.0 ** -k * (1.0 + 0.05 * rng.random((5, 3))))
    return np.concatenate(out)


def _batch(halos, dev):
    p = np.concatenate(halos) + 20.0
    ps = np.concatenate([[0], np.cumsum([len(h) for h in halos])])
    return batch.DeviceBatch.from_arrays(*p.T, np.full(len(p), 1e8), np.full(len(p), 2), ps, dev)


@pytest.mark.parametrize("core", [257, 300, 5000])
@pytest.mark.parametrize("shells", [1, 2, 3, 4])
@pytest.mark.parametrize("others", [False, True], ids=["alone", "among_others"])
def test_capture_takes_what_the_stage_takes(cuda_device, core, shells, others):
    halos = [_nested(core, shells, 3 * shells)]
    if others:
        hb = synth.catalogue(seed=4, nhalo=3, nmin=60, nmax=3000)
        p = np.stack([hb.x, hb.y, hb.z], 1)
        halos = [p[:hb.pstart[1]] - p[0], *halos, p[hb.pstart[1]:hb.pstart[2]] - p[hb.pstart[1]]]
    db = _batch(halos, cuda_device)
    cfg = batch.stage_config()
    ctx = batch.Context(0)
    ref = batch.stage_run(ctx, db, cfg, batch.StageBuffers(db.n, 32, cuda_device, keep_phi=True))
    ref = {f: getattr(ref, f).cpu().numpy() for f in FIELDS}
    out = batch.StageBuffers(db.n, 32, cuda_device, keep_phi=True)
    g = batch.StageGraph(ctx, db, cfg, out)
    for f in FIELDS:
        getattr(out, f).zero_()
    torch.cuda.synchronize()
    assert not g.run()  # the replay fits the plan
    torch.cuda.synchronize()
    got = {f: getattr(out, f).cpu().numpy() for f in FIELDS}
    g.close()
    ctx.close()
    np.testing.assert_array_equal(got["nearindex"], ref["nearindex"])
    np.testing.assert_array_equal(got["dens_sph"], ref["dens_sph"])
    # float sums in no fixed order, as between two runs of the stage
    assert np.abs(got["dens_mesh"] - ref["dens_mesh"]).max() <= 2e-6 * np.abs(ref["dens_mesh"]).max()
    np.testing.assert_allclose(got["phi"], ref["phi"], rtol=1e-6)
