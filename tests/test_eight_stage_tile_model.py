"""The CPU model of the stage groups' tile schedule (test_fused_stage_model.py) with the eight-cell halo
of the groups of eight: 112 output columns, tiles of 16, 32 and 48 rows."""
import numpy as np
import pytest

import test_fused_stage_model as model


@pytest.mark.parametrize("nx,ny", [(9, 40), (113, 33), (226, 49), (337, 97)])
@pytest.mark.parametrize("th", [16, 32, 48])
def test_eight_stage_schedule_equals_one_stage_at_a_time(monkeypatch, nx, ny, th):
    monkeypatch.setattr(model, "FH", 8)
    monkeypatch.setattr(model, "FOW", 112)
    rng = np.random.default_rng(nx * 1000 + ny * 10 + th)
    d1, d2, f0 = (rng.standard_normal((ny, nx)) for _ in range(3))
    sx, sy = rng.standard_normal(nx), rng.standard_normal(ny)
    coefs = [tuple(rng.uniform(-0.3, 0.3, 5)) for _ in range(8)]
    r2, r1 = model.one_stage_at_a_time(d1, d2, f0, coefs, sx, sy, 8)
    e2, e1 = model.tile_schedule(d1, d2, f0, coefs, sx, sy, 8, th, stand_in=1e300)
    assert np.array_equal(r1, e1) and np.array_equal(r2, e2)
