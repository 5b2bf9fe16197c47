"""CPU: the autotuner starts from the build that is shipped and leaves it only
for something faster."""
import json

import pytest

from galaxyfinder_b200 import build as B
from galaxyfinder_b200 import tune as T


def _tune(monkeypatch, tmp_path, params, ms, groups=("knn",)):
    """T.tune with stubbed builds: ms(parameters) is a variant's time."""
    import torch
    f = tmp_path / "tuned.json"
    if params is not None:
        f.write_text(json.dumps({"params": params}))
    monkeypatch.setattr(B, "TUNED", f)
    monkeypatch.setattr(B, "build", lambda *a, **k: None)
    monkeypatch.setattr(T, "build_variant", lambda src, p: p)
    monkeypatch.setattr(T, "measure", lambda p, nhalo, steps: {ph: ms(p) for _, ph in T.GROUPS.values()})
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda *a: "stub")
    return T.tune(64, 1, groups)["params"]


def _search_ms(p):
    """Networks 8.7 ms as shipped, 9.5 otherwise, the other searches 14.5."""
    if p["GF_KNN_ALGO"] != 3:
        return 14.5
    return 8.7 if (p["GF_KNNB_BLOCK"], p["GF_KNNB_MINB"], p["GF_KNNB_DYN"]) == (128, 6, 1) else 9.5


def test_keeps_the_shipped_search(monkeypatch, tmp_path):
    shipped = B.tuned_params()
    got = _tune(monkeypatch, tmp_path, shipped, _search_ms)
    assert {k: got[k] for k in shipped} == shipped


def test_finds_the_networks_without_a_record(monkeypatch, tmp_path):
    got = _tune(monkeypatch, tmp_path, None, _search_ms)
    assert got["GF_KNN_ALGO"] == 3


@pytest.mark.parametrize("groups", [("knn",), ("bh",), ("fft",), ("tsc",), ("tree",)])
def test_equal_times_change_nothing(monkeypatch, tmp_path, groups):
    shipped = B.tuned_params()
    got = _tune(monkeypatch, tmp_path, shipped, lambda p: 1.0, groups)
    assert {k: got[k] for k in shipped} == shipped


def test_network_candidates_fit_an_sm():
    """Shared memory (8576 bytes per warp, 1 KB per block of 228 KB) and threads."""
    base = dict(T.DEFAULTS, **B.tuned_params())
    assert base["GF_KNN_ALGO"] == 3
    seen = 0
    for stage in T.stages("knn"):
        for p in [base] + [dict(base, **ov) for ov in stage(base)]:
            if p["GF_KNN_ALGO"] == 3:
                b, m = p["GF_KNNB_BLOCK"], p["GF_KNNB_MINB"]
                assert b * m <= 2048 and m * (b // 32 * 8576 + 1024) <= 228 * 1024
                seen += p != base
            elif p["GF_KNN_ALGO"] == 2:  # heaps: see test_tuning.py
                warp = 32 * 32 * 8 + p["GF_KNNB_WIN"] * 48 + 32 * 16 + 32 * 4 + 32 * p["GF_KNNB_QUEUE"] * 8
                assert p["GF_KNNB_MINB"] * (p["GF_KNNB_BLOCK"] // 32 * warp + 1024) <= 228 * 1024
    assert seen >= 4
