"""Single projections take their scratch from a pool that keeps it between
calls: calls of several threads on streams of their own, and calls without a
wait between them, do not meet in it.
"""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [1, 4])
def test_calls_do_not_share_scratch(engine, threads):
    import torch

    G = engine.FanGeometry.covering
    plans = [engine.Plan.fan(G(64, 6.0, 90, 128)), engine.Plan.fan(G(200, 1.9, 150, 280)),
             engine.Plan.cone(engine.ConeGeometry(nx=24, ny=24, nz=16, voxel_mm=4.0, nproj=30, ndx=24, ndy=32,
                                                  pitch_mm=8.0, sod_mm=600.0, sdd_mm=1000.0))]
    rng = np.random.default_rng(2)
    cases = []
    for p in plans:
        img, sino = (torch.tensor(rng.random(s, dtype=np.float32), device="cuda") for s in (p.img_shape, p.sino_shape))
        cases.append((p, img, sino, torch.tensor(p.forward(img.cpu().numpy())), torch.tensor(p.back(sino.cpu().numpy()))))
    bad = []

    def work():
        st = torch.cuda.Stream()
        for rep in range(6):
            outs = []
            for p, img, sino, wf, wb in cases:
                f, b = torch.empty(p.sino_shape, device="cuda"), torch.empty(p.img_shape, device="cuda")
                st.wait_stream(torch.cuda.current_stream())
                p.forward_dev(img.data_ptr(), f.data_ptr(), st.cuda_stream)
                p.back_dev(sino.data_ptr(), b.data_ptr(), st.cuda_stream)
                outs.append((f, b, wf, wb))
            st.synchronize()
            bad.extend(1 for f, b, wf, wb in outs if not (torch.equal(f.cpu(), wf) and torch.equal(b.cpu(), wb)))

    pool = [threading.Thread(target=work) for _ in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    assert not bad
