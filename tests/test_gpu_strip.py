"""The back projector along lines where its strips, cells and ranges of views
end: images around the sizes of a cell (16 rows, 128 columns) and of a strip
(512 columns for a scan alone, 256 for groups), views around a block of 64,
detectors far finer and coarser than the pixels, against the FP64 oracle; and
every form and division of the work against one scan alone, bit for bit.

Tolerance: the rel-L2 of 1e-5 that all projectors are held to.  A ray's
crossing of a row is known to half an ulp of n/2 rows, 1.5e-5 at 512, so a
term of some 0.6 pixels to 2.5e-5, and a pixel adds up 24 terms and more of
independent errors: 5e-6.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


@pytest.mark.parametrize("n,views,dets", [
    (8, 24, 16), (15, 63, 40), (17, 64, 34), (127, 65, 160), (129, 24, 400), (255, 40, 300), (257, 33, 280),
    (512, 24, 640), (513, 30, 700), (64, 48, 1200), (200, 40, 50),
])
def test_strip_edges(engine, oracle, n, views, dets):
    g = engine.FanGeometry.covering(n, 384.0 / n, views, dets)
    p = engine.Plan.fan(g)
    rng = np.random.default_rng(n + views)
    sinos = [rng.random((views, dets)).astype(np.float32) for _ in range(5)]
    sinos[3][:] = 0.0  # a member with nothing to add
    alone = [p.back(s) for s in sinos]
    assert rel_l2(alone[0], oracle.fan_AT(oracle.fan_from_engine(g), sinos[0].astype(np.float64))) <= TOL
    assert not alone[3].any()
    for k in (1, 2, 3, 4, 5):  # pairs, threes, fours, and a scan beside a four
        ps = engine.ProjSet([p] * k)
        for got, want in zip(ps.back(sinos[:k]), alone):
            np.testing.assert_array_equal(got, want)
        ps.close()
    # many scans: other divisions of the views among CTAs
    ps = engine.ProjSet([p] * 24)
    for m, got in enumerate(ps.back([sinos[m % 5] for m in range(24)])):
        np.testing.assert_array_equal(got, alone[m % 5])
    ps.close()
    # the walk over tile runs is the same projection
    p.set_back_variant(0)
    assert rel_l2(p.back(sinos[0]), alone[0]) <= TOL


def test_no_ray_is_a_line(engine):
    """Rays that miss the grid and rays that end inside it."""
    n = 16
    e = np.zeros((2, 4, 4))
    e[0] = [-50.0, 100.0, 80.0, 100.0]  # past the grid
    e[1] = [8.0, -20.0, 8.2, 5.0]       # into it
    for frac, g in ((0, e[:1]), (1, e)):
        p = engine.Plan.rays(engine.RayGeometry(n, 1.0, len(g), 4, g.reshape(-1, 4)))
        out = p.back(np.ones((len(g), 4), np.float32))
        np.testing.assert_array_equal(out, engine.ProjSet([p, p]).back([np.ones((len(g), 4), np.float32)] * 2)[1])
        assert bool(out.any()) == bool(frac)


def test_mixed_batch(engine):
    """Plans that go by strips, by tile runs and by the table in one set."""
    G = engine.FanGeometry.covering
    a, b, c = engine.Plan.fan(G(100, 3.0, 130, 140)), engine.Plan.fan(G(72, 4.0, 65, 96)), engine.Plan.fan(G(48, 6.0, 60, 64))
    b.set_back_variant(0)
    c.set_back_variant(3)
    f = engine.Plan.fan(G(80, 4.0, 70, 100), alpha="fp32")
    plans = [a, b, a, c, f, a, b, c, f, a, a]
    rng = np.random.default_rng(5)
    sinos = [rng.standard_normal(p.sino_shape).astype(np.float32) for p in plans]
    ps = engine.ProjSet(plans)
    for _ in range(2):
        for p, s, got in zip(plans, sinos, ps.back(sinos)):
            np.testing.assert_array_equal(got, p.back(s))
