"""The search counters of a small batch are those of 32 queries per warp (a
search of few queries gives each of them several lanes, and a warp then tests
the same particles for fewer queries)."""
import pytest

from galaxyfinder_b200 import _lib, batch, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("npart", [120, 500])
def test_particle_tests_of_a_bucket(cuda_device, npart):
    """32 queries of one halo start with k = 32 of its particles and test each
    of the others at most once."""
    hb = synth.catalogue(seed=6, nhalo=1, nmin=npart, nmax=npart)
    db = batch.DeviceBatch.from_halobatch(hb)
    ctx = batch.Context(0)
    _, st = batch.stage_run(ctx, db, batch.stage_config(count_work=True), stats=True)
    ctx.close()
    assert _lib.tuning_value("GF_KNN_ALGO") == 3
    buckets = (hb.n + 31) // 32
    assert 0 < st["knn_batches"] <= buckets * (hb.n - 32)
