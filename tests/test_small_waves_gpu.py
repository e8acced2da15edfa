"""Renderers of few paths a wave on scenes of many photons a path: a wave never holds more photons than records.

16 spotlights of 16 photons make 256 a shading point, more than the records of 32 paths of a small renderer.
Every path's photons are the same whatever the waves, so the frame is a large renderer's up to the order of its
sums (fewer than 1,000 terms a channel: 1,000 * 2^-24 = 6e-5)."""
import numpy as np
import pytest
import torch

import dumbray_gb300 as dr
from dumbray_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lights,samples", [(16, 16), (4, 16), (5, 3), (1, 1)])
@pytest.mark.parametrize("wave", [1, 33, 1000, 4096])
@pytest.mark.parametrize("batch", [False, True])
def test_small_renderers_equal_a_large_one(cuda, lights, samples, wave, batch):
    rng = np.random.default_rng(lights)
    at = rng.uniform(-0.6, 0.6, (lights, 3)) * (1.0, 0.0, 1.0) + (0.0, 0.7, 0.0)
    spots = [dr.spotlight((1.0, 0.9, 0.8), 50.0, tuple(float(x) for x in p), (0.0, -1.0, 0.0), samples=samples, falloff_angle=160.0) for p in at]
    tris = np.concatenate([scenes.box((2.0, 2.0, 2.0), inward=True), scenes.icosphere(2, 0.4, (0.0, -0.4, 0.2))])
    sc = dr.Scene(tris, materials=[dr.dumb_based(diffuse=(0.7, 0.6, 0.5), metal=0.0)], lights=spots)
    cam = dr.camera(dr.LENS_SIMPLE_STOCHASTIC, position=(0.0, -0.2, -0.95), angle=60.0)
    params = dr.render_params(8, 16, dr.MODE_REFERENCE, samples=(1, 1), max_bounces=1, seed=3)
    frames = []
    for size in (1 << 16, wave):
        fb = dr.new_frame_buffer(8, 16, cuda)
        r = dr.Renderer(size)
        if batch:
            dr.Batch([(sc, cam, params, fb, 0, 1)]).render(r)
        else:
            r.render_blocks(sc, cam, fb, 0, 1, params)
        torch.cuda.synchronize()
        frames.append(fb)
    assert torch.allclose(*frames, rtol=6e-5, atol=1e-6)
    assert (frames[0][:, :3] > 0).any()
