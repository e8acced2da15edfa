"""Sums of the adjoint's gradients: a call adds to what the arrays hold, whatever the renderer served before.

By linearity a call over all blocks adds the sum of the calls over each block.  A component collects fewer
than 1e4 terms here, each positive, so a float32 sum of them in any order is within 1e4 * 2^-24 = 6e-4 of it."""
import numpy as np
import pytest
import torch

import dumbray_gb300 as dr
from dumbray_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(level):
    """A room whose ceiling quad emits; level < 0: no sphere."""
    parts = [scenes.box((2.0, 2.0, 2.0), inward=True), scenes.quad((0.0, 0.99, 0.0), (0.5, 0.5), (0.0, -1.0, 0.0))]
    if level >= 0:
        parts.append(scenes.icosphere(level, radius=0.6))
    tris = np.concatenate(parts)
    rng = np.random.default_rng(4)
    emission = np.zeros((len(tris), 3), np.float32)
    emission[12:14] = (5.0, 0.0, 3.0)
    sc = dr.Scene(tris, materials=[dr.lambert()], box_epsilon=dr.PHYSICAL_TREE)
    sc.set_triangle_params(rng.uniform(0.1, 0.9, (len(tris), 3)).astype(np.float32), emission, np.full(len(tris), 0.2, np.float32))
    return sc


@pytest.mark.parametrize("levels", [(-1, 3), (3, -1, 3)])   # the sums grow; shrink and come back
@pytest.mark.parametrize("width,height,depth", [(8, 16, 1), (33, 17, 3)])
def test_gradients_add_up_over_blocks(cuda, levels, width, height, depth):
    r = dr.Renderer(1 << 14)
    cam = dr.camera(dr.LENS_PINHOLE, position=(0.0, 0.0, -0.97), angle=60.0)
    params = dr.render_params(width, height, dr.MODE_PHYSICAL, samples=(2, 1), max_bounces=depth, seed=9)
    nb = dr.block_count(width, height)
    dl = dr.new_frame_buffer(width, height, cuda)
    dl[:, :3] = torch.rand((len(dl), 3), generator=torch.Generator(cuda).manual_seed(1), device=cuda) + 0.1
    for level in levels:
        sc = _scene(level)
        held = torch.rand((2, sc.n, 3), generator=torch.Generator(cuda).manual_seed(2), device=cuda)
        got = held.clone()
        r.render_adjoint(sc, cam, dl, 0, nb, params, got[0], got[1])
        want = held.double()
        for b in range(nb):
            part = torch.zeros_like(held)
            r.render_adjoint(sc, cam, dl, b, b + 1, params, part[0], part[1])
            want += part.double()
        assert torch.allclose(got.double(), want, rtol=6e-4, atol=6e-8)


def test_renderers_on_two_streams_add_to_the_same_arrays(cuda):
    sc = _scene(3)
    cam = dr.camera(dr.LENS_PINHOLE, position=(0.0, 0.0, -0.97), angle=60.0)
    width, height, rounds = 64, 64, 6
    params = dr.render_params(width, height, dr.MODE_PHYSICAL, samples=(1, 1), max_bounces=2, seed=9)
    nb = dr.block_count(width, height)
    dl = dr.new_frame_buffer(width, height, cuda) + 0.5
    renderers, streams = [dr.Renderer(1 << 14) for _ in range(2)], [torch.cuda.Stream() for _ in range(2)]
    got, one = torch.zeros((2, sc.n, 3), device=cuda), torch.zeros((2, sc.n, 3), device=cuda)
    renderers[0].render_adjoint(sc, cam, dl, 0, nb, params, one[0], one[1])
    torch.cuda.synchronize()
    for _ in range(rounds):
        for r, s in zip(renderers, streams):
            r.render_adjoint(sc, cam, dl, 0, nb, params, got[0], got[1], stream=s)
    torch.cuda.synchronize()
    # 4,096 paths of up to 3 terms a component: either sum is within 12,288 * 2^-24 = 7.4e-4 of its value
    assert torch.allclose(got.double(), 2 * rounds * one.double(), rtol=1.5e-3, atol=1e-6)
