"""What a ray's traversal has besides its line, forward.

Pieces that the reference's loop leaves out at a ray's end are taken from the
line's sum again: whatever their pixels hold, infinities and NaN and values far
above all others among them, the ray does not see it.

Tolerance: rel-L2 of 1e-6 to the clean image's projection (a line walked again
adds up in another order), and the same bits in every form.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a = np.asarray(a, np.float64)
    b = np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300))


def cut_rays(engine, n, way, dets=8):
    """Rays (unit pixels) that cross from row y0 into the next 0.02 mm before
    they leave the grid, so that the last pixel's piece is left out; and the
    pixels that are left out, one a ray.  way: bit 0 towards lower x, bit 1
    along y, bit 2 steps to lower rows."""
    ends, last = np.empty((dets, 4)), []
    for d in range(dets):
        y0, slope = 2 + d, 0.11 + 0.05 * d
        a = lambda x: y0 + 1 + slope * (x - (n - 0.02))  # noqa: E731
        e = np.array([-10.0, a(-10.0), n + 10.0, a(n + 10.0)])
        px = np.array([n - 1, y0 + 1])
        if way & 4:
            e[1::2], px[1] = n - e[1::2], n - 1 - px[1]
        if way & 1:
            e[0::2], px[0] = n - e[0::2], n - 1 - px[0]
        if way & 2:
            e, px = e[[1, 0, 3, 2]], px[::-1]
        ends[d] = e
        last.append(tuple(int(i) for i in px))
    return engine.RayGeometry(n, 1.0, 1, dets, ends), last


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e30, 3.0e38])
@pytest.mark.parametrize("way", range(8))
def test_pieces_left_out_stay_out(engine, way, value):
    n = 40
    g, last = cut_rays(engine, n, way)
    p = engine.Plan.rays(g)
    pixels = [set(map(int, p.trace_ray(0, d)[0])) for d in range(8)]
    img = np.random.default_rng(way).random((n, n)).astype(np.float32)
    clean = p.forward(img)
    marked = img.copy()
    for d, (x, y) in enumerate(last):
        assert x * n + y not in pixels[d]  # left out, as meant
        marked[x, y] = value
    hits = np.array([any(x * n + y in pixels[d] for x, y in last) for d in range(8)])
    assert not hits.all()
    forms = [p.forward(marked)]
    for k in (2, 3, 4):
        ps = engine.ProjSet([p] * k)
        forms += ps.forward([marked] + [img] * (k - 1))[:1]
        ps.close()
    p.set_forward_variant(2, 16, 16)
    forms.append(p.forward(marked))
    for got in forms:
        assert np.all(np.isfinite(got[0][~hits]))
        assert rel_l2(got[0][~hits], clean[0][~hits]) <= 1e-6
        np.testing.assert_array_equal(got, forms[0])


def test_only_the_piece_left_out_is_there(engine):
    """An image that holds nothing else projects to nothing."""
    n = 40
    g, last = cut_rays(engine, n, 0)
    p = engine.Plan.rays(g)
    img = np.zeros((n, n), np.float32)
    img[last[3]] = 7.0
    want = np.array([last[3][0] * n + last[3][1] in p.trace_ray(0, d)[0] for d in range(8)])
    np.testing.assert_array_equal(p.forward(img)[0] != 0.0, want)
