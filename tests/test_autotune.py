"""The autotuner's search without a GPU: a stand-in for the timed contexts."""
import pytest

from pfem2_b200 import _abi as A
from pfem2_b200 import autotune


@pytest.mark.parametrize("cluster", [False, True])
def test_velocity_shapes_not_searched_stay_automatic(monkeypatch, cluster):
    """a search of the particle shapes neither times its candidates with the
    velocity shapes of the first context nor writes them: contexts of one key
    differ in size by up to a factor of two, and small ones solve in one
    cluster, which any velocity shape rules out"""
    resolved = dict.fromkeys(A.TUNING_FIELDS, 0)
    resolved.update(advect_blocks_per_sm=16, advect_split=2, rebin_blocks_per_sm=8, p_blocks_per_sm=1)
    if not cluster:
        resolved.update(vel_tile_slices=3, vel_blocks_per_sm=1)
    asked = []

    def fake_measure(specs, tuning, steps, warmup, prepare=None, **kw):
        asked.append(dict(tuning or {}))
        return 1.0 + len(asked) % 3, dict(resolved, **{k: v for k, v in (tuning or {}).items() if v})

    class FakeSolver:
        def __init__(self, *a, **k):
            pass

        def tuning_key(self):
            return "DEV 2 4 12 0"

        def close(self):
            pass

    monkeypatch.setattr(autotune, "measure", fake_measure)
    monkeypatch.setattr(autotune, "Solver", FakeSolver)
    res = autotune.tune([None], space={"advect_blocks_per_sm": [8, 16], "rebin_blocks_per_sm": [4, 8]}, steps=1, warmup=0)
    for t in asked + [res["tuning"]]:
        assert not t.get("vel_tile_slices") and not t.get("vel_blocks_per_sm")
    assert res["tuning"]["advect_blocks_per_sm"] in (8, 16)
