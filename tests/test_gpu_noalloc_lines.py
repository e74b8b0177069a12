"""The forward projection that allocates nothing, on plans whose rays are walked
as lines: it costs what the projection costs, and a launch whose CTAs' partial
sums would not fit its array takes larger CTAs.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def buffers(p, seed=0):
    import torch

    rng = np.random.default_rng(seed)
    img, g = (torch.tensor(rng.random(s, dtype=np.float32), device="cuda") for s in (p.img_shape, p.sino_shape))
    return img, g, torch.empty(p.sino_shape, device="cuda"), torch.zeros(1, dtype=torch.float64, device="cuda")


def residual(engine, p, bufs, stream):
    rc = engine.lib().at_forward_residual_noalloc(p.handle, *(b.data_ptr() for b in bufs), stream)
    assert rc == 0, engine.lib().at_last_error().decode()


@pytest.mark.parametrize("n,views,dets", [(16, 4096, 1200), (64, 2731, 1500)])
def test_many_rays_take_larger_ctas(engine, n, views, dets):
    import torch

    p = engine.Plan.fan(engine.FanGeometry.covering(n, 384.0 / n, views, dets))
    bufs = buffers(p)
    for _ in range(2):
        residual(engine, p, bufs, None)
        torch.cuda.synchronize()
        img, g, r, energy = (b.cpu().numpy() for b in bufs)
        np.testing.assert_array_equal(r, g - p.forward(img))
        want = float(np.sum(r.astype(np.float64) ** 2))
        assert abs(energy[0] - want) <= 1e-12 * want


@pytest.mark.parametrize("n,views,dets", [(512, 720, 888), (1024, 60, 1536)])
def test_costs_what_the_projection_costs(engine, n, views, dets):
    """Best of several runs of twenty calls against the projection's: the
    residual's extra reads and its sum are a few per cent, the two extra copies
    of a few bytes some microseconds; walking the image itself took 3.5 times
    as long."""
    import torch

    p = engine.Plan.fan(engine.FanGeometry.covering(n, 384.0 / n, views, dets))
    bufs = buffers(p)
    out = torch.empty(p.sino_shape, device="cuda")
    st = torch.cuda.Stream()

    def best(call):
        times = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(st)
            for _ in range(20):
                call()
            b.record(st)
            b.synchronize()
            times.append(a.elapsed_time(b))
        return min(times)

    torch.cuda.synchronize()
    plain = best(lambda: p.forward_dev(bufs[0].data_ptr(), out.data_ptr(), st.cuda_stream))
    assert best(lambda: residual(engine, p, bufs, st.cuda_stream)) <= 1.6 * plain
