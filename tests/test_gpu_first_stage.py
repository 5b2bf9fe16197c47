"""The first stage of a new context on a small batch runs on the context's own
stream alone: the side streams, which cost more to make than they save there,
come with its second stage, or with a first one of 32,768 particles."""
import json

import numpy as np
import pytest
import torch

from galaxyfinder_b200 import _lib, batch, synth

pytestmark = pytest.mark.gpu

FIELDS = ("nearindex", "dens_sph", "dens_mesh", "penergy", "phi")


def _streams(path, call):
    """The number of streams whose kernels `call` runs."""
    acts = [torch.profiler.ProfilerActivity.CPU, torch.profiler.ProfilerActivity.CUDA]
    with torch.profiler.profile(activities=acts) as prof:
        call()
        torch.cuda.synchronize()
    prof.export_chrome_trace(str(path))
    events = json.loads(path.read_text())["traceEvents"]
    used = {e["args"]["stream"] for e in events if e.get("cat") == "kernel"}
    assert used
    return len(used)


@pytest.mark.parametrize("npart,want", [(120, (1, 3, 3)), (32767, (1, 3, 3)), (32768, (3, 3, 3))])
def test_streams_of_the_first_stages(cuda_device, tmp_path, npart, want):
    hb = synth.catalogue(seed=3, nhalo=1, nmin=npart + 8, nmax=npart + 8)
    db = batch.DeviceBatch.from_arrays(*(a[:npart] for a in (hb.x, hb.y, hb.z, hb.mass, hb.type)), [0, npart])
    cfg = batch.stage_config()
    ctx = batch.Context(0)
    outs, used = [], []
    for i in range(3):
        o = batch.StageBuffers(npart, 32, cuda_device, keep_phi=True)
        used.append(_streams(tmp_path / f"{i}.json", lambda: batch.stage_run(ctx, db, cfg, o)))
        outs.append({f: getattr(o, f).cpu().numpy() for f in FIELDS})
    ctx.close()
    assert tuple(used) == want
    for o in outs[1:]:  # float sums in no fixed order, as between two runs
        np.testing.assert_array_equal(o["nearindex"], outs[0]["nearindex"])
        np.testing.assert_array_equal(o["dens_sph"], outs[0]["dens_sph"])
        assert np.abs(o["dens_mesh"] - outs[0]["dens_mesh"]).max() <= 2e-6 * outs[0]["dens_mesh"].max()
        np.testing.assert_allclose(o["phi"], outs[0]["phi"], rtol=1e-6)
        # phi * potentfact + the background term, rounded once; of opposite signs
        assert np.abs(o["penergy"] - outs[0]["penergy"]).max() <= 2e-6 * np.abs(outs[0]["penergy"]).max()


def test_streams_of_two_priorities(cuda_device, tmp_path):
    """A context switched between streams of two priorities makes no streams
    for either (after a first small stage) until a priority comes twice."""
    hb = synth.catalogue(seed=3, nhalo=4, nmin=100, nmax=2000)
    db = batch.DeviceBatch.from_halobatch(hb)
    cfg = batch.stage_config()
    ctx = batch.Context(0)
    used = []
    for i, prio in enumerate((0, -1, 0, -1, -1, 0, -1)):
        s = torch.cuda.Stream(priority=prio)
        _lib.check(_lib.lib().gf_ctx_set_stream(ctx.handle, _lib.ctypes.c_void_p(s.cuda_stream)))
        o = batch.StageBuffers(hb.n, 32, cuda_device)
        torch.cuda.synchronize()
        used.append(_streams(tmp_path / f"{i}.json", lambda: batch.stage_run(ctx, db, cfg, o)))
    ctx.close()
    assert used == [1, 1, 1, 1, 3, 1, 3]
