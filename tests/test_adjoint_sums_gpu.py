"""Sums of the adjoint's gradients against renders.

The image is linear in every emitter and a sum of contributions that each carry one albedo factor per
path vertex; renders of the same seed with one bounce more add exactly the contributions with one
factor more.  So, for any dL/dI,
    sum(emission * grad_emission) = <dL/dI, image>
    sum(albedo * grad_albedo)     = sum over d of d <dL/dI, image_d - image_{d-1}>.
Every term is positive here, so float32 accumulation in any order stays within n ulp of the sum for
chains of n additions; blocks add at most some thousand terms to one sum and the global arrays some
thousand block sums: 4e3 * 2^-24 = 2.4e-4, on either side of the equation."""
import numpy as np
import pytest
import torch

import dumbray_gb300 as dr
from dumbray_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(level):
    """A room whose ceiling quad and some sphere triangles emit; level < 0: no sphere (every triangle is large)."""
    parts = [scenes.box((2.0, 2.0, 2.0), inward=True), scenes.quad((0.0, 0.99, 0.0), (0.5, 0.5), (0.0, -1.0, 0.0))]
    if level >= 0:
        parts.append(scenes.icosphere(level, radius=0.6))
    tris = np.concatenate(parts)
    rng = np.random.default_rng(4)
    albedo = rng.uniform(0.1, 0.9, (len(tris), 3)).astype(np.float32)
    emission = np.zeros((len(tris), 3), np.float32)
    emission[12:14] = 5.0
    if level >= 0:
        emission[14::97] = (3.0, 2.0, 1.0)
    sc = dr.Scene(tris, materials=[dr.lambert()], box_epsilon=dr.PHYSICAL_TREE)
    sc.set_triangle_params(albedo, emission, np.full(len(tris), 0.2, np.float32))
    return sc, albedo.astype(np.float64), emission.astype(np.float64)


@pytest.mark.parametrize("level", [-1, 2, 5])
@pytest.mark.parametrize("width,height,spp,depth", [(8, 16, 1, 1), (33, 17, 2, 3), (200, 136, 4, 5)])
def test_gradient_sums_equal_renders(cuda, level, width, height, spp, depth):
    sc, albedo, emission = _scene(level)
    cam = dr.camera(dr.LENS_PINHOLE, position=(0.0, 0.0, -0.97), angle=60.0)
    nb = dr.block_count(width, height)
    r = dr.Renderer(1 << 18)
    dl = dr.new_frame_buffer(width, height, cuda)
    dl[:, :3] = torch.rand((len(dl), 3), generator=torch.Generator(cuda).manual_seed(1), device=cuda) + 0.1
    share = []
    for d in range(depth + 1):
        fb = dr.new_frame_buffer(width, height, cuda)
        r.render_blocks(sc, cam, fb, 0, nb, dr.render_params(width, height, dr.MODE_PHYSICAL, samples=(spp, 1), max_bounces=d, seed=9))
        share.append(float((dl[:, :3].double() * fb[:, :3].double()).sum()))
    ga, ge = (torch.zeros((sc.n, 3), dtype=torch.float32, device=cuda) for _ in range(2))
    r.render_adjoint(sc, cam, dl, 0, nb, dr.render_params(width, height, dr.MODE_PHYSICAL, samples=(spp, 1), max_bounces=depth, seed=9), ga, ge)
    got_e = float((ge.double().cpu().numpy() * emission).sum())
    got_a = float((ga.double().cpu().numpy() * albedo).sum())
    want_a = sum(d * (share[d] - share[d - 1]) for d in range(1, depth + 1))
    assert got_e == pytest.approx(share[-1], rel=5e-4)
    assert got_a == pytest.approx(want_a, rel=5e-4, abs=5e-4 * share[-1])
