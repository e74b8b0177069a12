"""What a ray's traversal has besides its line, forward.

Pieces that the reference's loop leaves out at a ray's end are taken from the
line's sum again: whatever their pixels hold, infinities and NaN and values far
above all others among them, the ray does not see it.  Rays that are no lines
are sums over their own pixels, alone and beside rays that are, in every group
form.

Tolerance: rel-L2 of 1e-6 to the clean image's projection (a line walked again
adds up in another order), and the same bits in every form; the rel-L2 of 1e-5
to the FP64 oracle that all projectors are held to.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 1e-5


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

def inside(engine, n, views, dets, share, seed=3):
    """A fan whose rays end inside the grid, `share` of them."""
    base = engine.RayGeometry.fan_from_view_table(n, 384.0 / n, dets, np.arange(views) * 360.0 / views,
                                                  det_pitch_deg=61.0 / dets)
    rng = np.random.default_rng(seed)
    e = base.endpoints.copy()
    m = rng.random(len(e)) < share
    t, r = rng.random(m.sum()) * 2 * np.pi, 150 * np.sqrt(rng.random(m.sum()))
    e[m, 2:] = 192 + np.stack([r * np.cos(t), r * np.sin(t)], 1)
    return engine.RayGeometry(n, 384.0 / n, views, dets, e)


@pytest.mark.parametrize("n,views,dets,share", [(16, 9, 34, 0.1), (33, 20, 66, 0.05), (130, 40, 200, 0.03), (512, 12, 888, 0.05)])
def test_rays_that_end_inside(engine, oracle, n, views, dets, share):
    g = inside(engine, n, views, dets, share)
    p = engine.Plan.rays(g)
    rng = np.random.default_rng(n)
    imgs = [rng.standard_normal((n, n)).astype(np.float32) for _ in range(5)]
    alone = [p.forward(x) for x in imgs]
    assert rel_l2(alone[0], oracle.fan_A(oracle.fan_from_engine(g), imgs[0].astype(np.float64))) <= TOL
    for k in (2, 3, 4, 5):
        ps = engine.ProjSet([p] * k)
        for got, want in zip(ps.forward(imgs[:k]), alone):
            np.testing.assert_array_equal(got, want)
        ps.close()


def test_few_rays_that_end_inside_cost_little(engine):
    """One ray in twenty of 512^2, 360 x 888, against none of them (best of
    several runs of ten calls): their pixels are as many again as a twentieth
    of the others' and two loads each; a lane for each such ray took 2.8 times
    as long, the walk over segments 1.9."""
    import torch

    times = []
    for share in (0.0, 0.05):
        p = engine.Plan.rays(inside(engine, 512, 360, 888, share))
        img, out = torch.rand(512, 512, device="cuda"), torch.empty(p.sino_shape, device="cuda")
        st = torch.cuda.Stream()
        torch.cuda.synchronize()
        runs = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(st)
            for _ in range(10):
                p.forward_dev(img.data_ptr(), out.data_ptr(), st.cuda_stream)
            b.record(st)
            b.synchronize()
            runs.append(a.elapsed_time(b))
        times.append(min(runs))
    assert times[1] <= 1.9 * times[0]
