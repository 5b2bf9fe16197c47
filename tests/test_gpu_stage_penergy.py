"""The stage's energies (potential and background term, which is prepared on a
side stream ahead of the search) with its parts side by side, one after the
other and replayed; every output is overwritten between two runs."""
import numpy as np
import pytest
import torch

from galaxyfinder_b200 import batch, synth

pytestmark = pytest.mark.gpu

FIELDS = ("nearindex", "dens_sph", "dens_mesh", "penergy", "phi")


def _get_and_clear(out):
    torch.cuda.synchronize()
    got = {f: getattr(out, f).cpu().numpy() for f in FIELDS}
    for f in FIELDS:
        getattr(out, f).fill_(-77)
    torch.cuda.synchronize()
    return got


@pytest.mark.parametrize("nhalo,nmin,nmax", [(1, 120, 120), (60, 40, 4000), (2, 45000, 65000)])
@pytest.mark.parametrize("add_bg", [True, False])
def test_energies_side_by_side(cuda_device, nhalo, nmin, nmax, add_bg):
    hb = synth.catalogue(seed=nhalo, nhalo=nhalo, nmin=nmin, nmax=nmax)
    db = batch.DeviceBatch.from_halobatch(hb)
    cfg = batch.stage_config(add_bg=add_bg)
    ctx = batch.Context(0)
    out = batch.StageBuffers(hb.n, 32, cuda_device, keep_phi=True)
    batch.stage_run(ctx, db, cfg, out, stats=True)  # one after the other
    ref = _get_and_clear(out)
    # energies are phi * potentfact plus the background term in double, rounded
    # once: with phi within 1e-6 (node sums in no fixed order) they are within
    # 1e-6 of the potential's part and a unit in the last place
    factor = np.median((ref["penergy"] / ref["phi"].astype(np.float64))) if not add_bg else _factor(ctx, db, out)
    part = np.abs(factor * ref["phi"].astype(np.float64))
    bar = 1e-6 * part + np.spacing(np.abs(ref["penergy"]))

    def check(got):
        np.testing.assert_array_equal(got["nearindex"], ref["nearindex"])
        np.testing.assert_array_equal(got["dens_sph"], ref["dens_sph"])
        assert np.abs(got["dens_mesh"] - ref["dens_mesh"]).max() <= 2e-6 * ref["dens_mesh"].max()
        assert (np.abs(got["phi"] - ref["phi"]) <= 1e-6 * np.abs(ref["phi"])).all()
        assert (np.abs(got["penergy"].astype(np.float64) - ref["penergy"]) <= bar).all()

    for _ in range(3):
        batch.stage_run(ctx, db, cfg, out)
        check(_get_and_clear(out))
    g = batch.StageGraph(ctx, db, cfg, out)
    check(_get_and_clear(out))
    for _ in range(2):
        assert not g.run()
        check(_get_and_clear(out))
    g.close()
    ctx.close()


def _factor(ctx, db, out):
    """potentfact, from a run without the background term."""
    batch.stage_run(ctx, db, batch.stage_config(add_bg=False), out, stats=True)
    got = _get_and_clear(out)
    return np.median(got["penergy"] / got["phi"].astype(np.float64))
