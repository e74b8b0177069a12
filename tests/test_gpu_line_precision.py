"""The projectors along lines are no further from 64 bits than the walks over the
traversal's segments were, down to the smallest grids.

A ray's next crossing is a running sum, whose rounding counts beside the
pixels' size on small grids and beside that of the ray's own place on large
ones.  Limits: the mean error of the walk by decision bits (forward) and of the
tile runs (back), which the lines replaced, over sinograms and phantoms of these
sizes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIMITS = {  # forward of a phantom, of noise; back of its sinogram, of noise
    (16, 40, 32): (1.48e-7, 9.92e-8, 1.12e-7, 1.10e-7),
    (32, 48, 64): (1.88e-7, 1.18e-7, 1.46e-7, 1.40e-7),
    (48, 60, 96): (2.09e-7, 1.44e-7, 1.92e-7, 1.87e-7),
    (64, 90, 128): (2.07e-7, 1.46e-7, 1.92e-7, 1.88e-7),
    (128, 90, 256): (2.12e-7, 1.94e-7, 2.77e-7, 2.64e-7),
}


def rel_l2(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n,views,dets", sorted(LIMITS))
def test_error_against_64_bits(engine, oracle, n, views, dets):
    g = engine.FanGeometry.covering(n, 384.0 / n, views, dets)
    p, fan = engine.Plan.fan(g), oracle.fan_from_engine(g)
    errors = []
    for seed in range(4):
        rng = np.random.default_rng(seed)
        img = [engine.phantom.ellipse_phantom(n, seed=seed, n_random=8).astype(np.float32),
               rng.random((n, n), dtype=np.float32)]
        clean = oracle.fan_A(fan, img[0].astype(np.float64))
        sino = [engine.phantom.poisson_sinogram(clean, 1e4, seed).astype(np.float32),
                rng.random((views, dets), dtype=np.float32)]
        errors.append([rel_l2(p.forward(x), oracle.fan_A(fan, x.astype(np.float64))) for x in img] +
                      [rel_l2(p.back(x), oracle.fan_AT(fan, x.astype(np.float64))) for x in sino])
    mean = np.mean(errors, axis=0)
    assert np.all(mean <= np.array(LIMITS[n, views, dets])), mean
