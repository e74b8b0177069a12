"""Single projections can be captured into a graph and replayed: every kind of
plan, both directions, and the call that allocates nothing; the replays give
the call's own result.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def plan(engine, kind):
    G = engine.FanGeometry.covering
    if kind == "fan":
        return engine.Plan.fan(G(96, 2.0, 100, 160))
    if kind == "runs":
        p = engine.Plan.fan(G(96, 2.0, 100, 160))
        p.set_back_variant(0)
        return p
    if kind == "fp32":
        return engine.Plan.fan(G(96, 2.0, 100, 160), alpha="fp32")
    if kind == "rays":
        return engine.Plan.rays(engine.RayGeometry.msbeam_parallel(64, 20, 96))
    if kind == "goldnc":
        return engine.Plan.goldnc()
    return engine.Plan.cone(engine.ConeGeometry(24, 24, 16, 1.0, 12, 16, 20, 1.5, 60.0, 110.0))


@pytest.mark.parametrize("kind", ["fan", "runs", "fp32", "rays", "cone", "goldnc"])
@pytest.mark.parametrize("call", ["forward", "back", "noalloc"])
def test_captured(engine, kind, call):
    import torch

    p = plan(engine, kind)
    rng = np.random.default_rng(1)
    img, sino = (torch.tensor(rng.random(s, dtype=np.float32), device="cuda") for s in (p.img_shape, p.sino_shape))
    out = torch.zeros(p.img_shape if call == "back" else p.sino_shape, device="cuda")
    energy = torch.zeros(1, dtype=torch.float64, device="cuda")

    def run(st):
        if call == "forward":
            p.forward_dev(img.data_ptr(), out.data_ptr(), st)
        elif call == "back":
            p.back_dev(sino.data_ptr(), out.data_ptr(), st)
        else:
            rc = engine.lib().at_forward_residual_noalloc(p.handle, img.data_ptr(), sino.data_ptr(), out.data_ptr(),
                                                          energy.data_ptr(), st)
            assert rc == 0, engine.lib().at_last_error().decode()

    if call == "noalloc":  # (its first call on a device is made before a capture)
        run(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(torch.cuda.current_stream().cuda_stream)
    replays = []
    for _ in range(3):
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        replays.append(out.clone())
    run(torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert bool(out.any())
    for r in replays:
        assert torch.equal(r, out)
