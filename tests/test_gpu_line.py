"""Projectors that take each ray as a line through the grid, against the FP64
oracle's traversal, where the two could part: ray tables whose rays end inside
the grid, run along grid lines or the image's edges or across the diagonal,
miss it, come in any order and direction, and pixels so small that the
reference leaves several of a ray's last ones out; and grids around the blocks
of 32 rows that the walk works in.

Images and sinograms are noise, so every pixel and ray counts.  Tolerance: the
rel-L2 of 1e-5 that all projectors are held to (for noise the sums are a few
hundred terms of one sign, each exact to about 1e-7).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def table(engine, n, px, seed, views=9, dets=70):
    """Views of rays all round: straight through at random angles and offsets
    (sorted, reversed and shuffled), along grid lines and edges, diagonals,
    and a view whose rays end inside the grid."""
    rng = np.random.default_rng(seed)
    half = n * px / 2
    e = np.empty((views, dets, 4))
    for v in range(views):
        a = rng.uniform(0, 2 * np.pi)
        off = np.sort(rng.uniform(-0.75, 0.75, dets)) * n * px
        if v == 1:
            a, off = 0.0, (np.arange(dets) - dets // 2) * px  # on grid lines
        if v == 2:
            a, off = np.pi / 2, (np.arange(dets) - dets // 2 + 0.25) * px
        if v == 3:
            a, off = np.pi / 4, (np.arange(dets) - dets // 2) * px * np.sqrt(0.5)
        if v == 4:
            off = off[::-1]
        if v == 5:
            off = rng.permutation(off)
        u = np.array([np.cos(a), np.sin(a)])
        w = np.array([-u[1], u[0]])
        for d in range(dets):
            c = half + off[d] * w
            r = 2.0 * n * px
            s, t = c - r * u, c + r * u
            if v == 6 and d % 7 == 0:
                t = half + rng.uniform(-0.4, 0.4, 2) * n * px
            e[v, d] = (*s, *t)
    return engine.RayGeometry(n, px, views, dets, e.reshape(-1, 4))


@pytest.mark.parametrize("n,px", [(8, 1.0), (31, 0.7), (32, 1.0), (33, 2.0), (64, 0.03), (97, 0.01)])
def test_ray_tables(engine, oracle, n, px):
    g = table(engine, n, px, seed=n)
    p, fan = engine.Plan.rays(g), oracle.fan_from_engine(g)
    rng = np.random.default_rng(n + 1)
    img = rng.random((n, n)).astype(np.float32)
    sino = rng.random(p.sino_shape).astype(np.float32)
    assert rel_l2(p.forward(img), oracle.fan_A(fan, img.astype(np.float64))) <= TOL
    assert rel_l2(p.back(sino), oracle.fan_AT(fan, sino.astype(np.float64))) <= TOL
    for k in (2, 4):  # groups: the same sums
        ps = engine.ProjSet([p] * k)
        for got, want in ((ps.forward([img * (m + 1) for m in range(k)]), [p.forward(img * (m + 1)) for m in range(k)]),
                          (ps.back([sino * (m + 1) for m in range(k)]), [p.back(sino * (m + 1)) for m in range(k)])):
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
        ps.close()


@pytest.mark.parametrize("n,views,dets", [(8, 1, 2), (31, 3, 66), (32, 17, 64), (33, 16, 62), (65, 33, 130),
                                          (127, 65, 258), (40, 48, 400)])
def test_fan_noise(engine, oracle, n, views, dets):
    g = engine.FanGeometry.covering(n, 300.0 / n, views, dets)
    p, fan = engine.Plan.fan(g), oracle.fan_from_engine(g)
    rng = np.random.default_rng(n)
    img = rng.random((n, n)).astype(np.float32)
    sino = rng.random(p.sino_shape).astype(np.float32)
    assert rel_l2(p.forward(img), oracle.fan_A(fan, img.astype(np.float64))) <= TOL
    assert rel_l2(p.back(sino), oracle.fan_AT(fan, sino.astype(np.float64))) <= TOL


def test_infinite_pixels_stay_on_their_rays(engine, oracle):
    """An infinite pixel reaches exactly the rays that cross it (as a sum that
    is not finite: the compensated sums make it NaN)."""
    g = engine.FanGeometry.covering(64, 2.0, 40, 128)
    p, fan = engine.Plan.fan(g), oracle.fan_from_engine(g)
    img = np.random.default_rng(1).random((64, 64)).astype(np.float32)
    mark = np.zeros((64, 64))
    mark[17, 40] = 1.0
    hit = oracle.fan_A(fan, mark)
    clean = p.forward(img)
    img[17, 40] = np.inf
    got = p.forward(img)
    np.testing.assert_array_equal(got[hit == 0], clean[hit == 0])
    assert not np.any(np.isfinite(got[hit > 1e-3]))
