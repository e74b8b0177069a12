"""A pinned back projector can be unpinned: the plan is then a fresh one again,
bit for bit, alone and in groups, and says which form it is in.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mask", [0, 1, 2, 3])
def test_pin_and_reset(engine, mask):
    g = engine.FanGeometry.covering(130, 2.0, 100, 180)
    p, fresh = engine.Plan.fan(g), engine.Plan.fan(g)
    rng = np.random.default_rng(mask)
    sinos = [rng.standard_normal(p.sino_shape).astype(np.float32) for _ in range(3)]
    want = [fresh.back(s) for s in sinos]
    assert p.back_variant == fresh.back_variant == -1
    p.set_back_variant(mask)
    assert p.back_variant == mask
    assert not np.array_equal(p.back(sinos[0]), want[0])  # crossings rounded otherwise
    p.reset_back_variant()
    assert p.back_variant == -1
    assert p.stats["bp_table_use"] == 0
    for s, w in zip(sinos, want):
        np.testing.assert_array_equal(p.back(s), w)
    ps = engine.ProjSet([p, p, p])
    for got, w in zip(ps.back(sinos), want):
        np.testing.assert_array_equal(got, w)
    ps.close()


def test_plans_without_lines(engine):
    p = engine.Plan.fan(engine.FanGeometry.covering(64, 4.0, 60, 96), alpha="fp32")
    assert p.back_variant == 0
    p.set_back_variant(1)
    assert p.back_variant == 1
    p.reset_back_variant()
    assert p.back_variant == 0
    cone = engine.Plan.cone(engine.ConeGeometry(24, 24, 16, 1.0, 12, 16, 20, 1.5, 60.0, 110.0))
    for call in (cone.reset_back_variant, lambda: cone.back_variant):
        with pytest.raises(engine.AtError):
            call()
