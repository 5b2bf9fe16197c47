"""The phase times of a timed stage: planning the smoothing (filter tables of
long axes, made on the host) is part of the mesh phases, not of the recentring."""
import numpy as np
import pytest

from galaxyfinder_b200 import _lib, batch

pytestmark = pytest.mark.gpu


def test_mesh_planning_is_no_recentring(cuda_device):
    """A filament: the x axis by the reference's rule has some 2600 cells, whose
    n^2 filter sums take the host several times as long as every kernel of the
    recentring, a few microseconds each."""
    rng = np.random.default_rng(1)
    n = 3000
    p = rng.random((n, 3)) * [10.4, 0.05, 0.05] + 5.0
    db = batch.DeviceBatch.from_arrays(*p.T, np.full(n, 1e8), np.full(n, 2), [0, n], cuda_device)
    cfg = batch.stage_config(mesh=batch.mesh_rule(mode=_lib.MESH_REFERENCE))
    ctx = batch.Context(0)
    times = []
    for _ in range(5):
        _, st = batch.stage_run(ctx, db, cfg, stats=True)
        times.append((st["ms_recentre"], st["ms_tsc"] + st["ms_smooth"]))
    ctx.close()
    recentre, mesh = np.min(times, axis=0)
    assert mesh > 2.0 and recentre < 0.5 * mesh
