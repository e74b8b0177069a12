"""The back projector along lines keeps its 32-bit sums in range on ray tables.

Rays of one view meet in a pixel within the last 0.05 mm of the grid.  The
reference's loop leaves those last pieces out, so no count of the traversal's
segments sees the pixel, but the lines run through it.  Sums past 2^31 would
put the image off by whole multiples of 2^32 quanta.

Tolerance: the rel-L2 of 1e-5 that all projectors are held to; an overflow is
of order one.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def fan_into(engine, n, px, inside, dets, edge):
    """Rays of one view fanned over 1.4 rad through the middle of a pixel
    `inside` pixels from the edge that they leave the grid by."""
    ext = n * px
    focus = np.array([ext - (inside + 0.5) * px, (n // 2 + 0.5) * px])
    t = np.linspace(-0.7, 0.7, dets)
    u = np.stack([np.cos(t), np.sin(t)], 1)
    s, d = focus - 4 * ext * u, focus + 4 * ext * u
    if edge % 2:  # the same towards lower coordinates
        s, d = ext - s, ext - d
    if edge >= 2:  # along y
        s, d = s[:, ::-1], d[:, ::-1]
    return engine.RayGeometry(n, px, 1, dets, np.concatenate([s, d], 1))


@pytest.mark.parametrize("edge", range(4))
@pytest.mark.parametrize("n,px,inside", [(512, 0.002, 10), (512, 0.005, 4), (256, 0.01, 2), (64, 0.05, 0), (64, 1.0, 3)])
def test_rays_that_meet_at_the_exit(engine, oracle, n, px, inside, edge):
    g = fan_into(engine, n, px, inside, 8192 if n > 64 else 2048, edge)
    p, fan = engine.Plan.rays(g), oracle.fan_from_engine(g)
    sino = np.ones(p.sino_shape, np.float32)
    want = oracle.fan_AT(fan, sino.astype(np.float64))
    got = p.back(sino)
    assert rel_l2(got, want) <= TOL
    ps = engine.ProjSet([p, p])
    for out in ps.back([sino, sino]):
        np.testing.assert_array_equal(out, got)
    ps.close()
