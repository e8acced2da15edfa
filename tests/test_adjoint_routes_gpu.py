"""The two ways a gradient term takes: padded sums of the call, or the caller's arrays (few paths, captured calls).

Terms are positive and fewer than 1e4 a component, so a float32 sum of them in any order is within
1e4 * 2^-24 = 6e-4 of it."""
import numpy as np
import pytest
import torch

import dumbray_gb300 as dr
from dumbray_gb300 import scenes

pytestmark = pytest.mark.gpu


def _scene(level):
    """A room whose ceiling quad emits, with a sphere; below 256 triangles at level 0, more than 1,024 at 3."""
    tris = np.concatenate([scenes.box((2.0, 2.0, 2.0), inward=True), scenes.quad((0.0, 0.99, 0.0), (0.5, 0.5), (0.0, -1.0, 0.0)),
                           scenes.icosphere(level, radius=0.6)])
    emission = np.zeros((len(tris), 3), np.float32)
    emission[12:14] = (5.0, 0.0, 3.0)
    sc = dr.Scene(tris, materials=[dr.lambert()], box_epsilon=dr.PHYSICAL_TREE)
    sc.set_triangle_params(np.full((len(tris), 3), 0.6, np.float32), emission, np.full(len(tris), 0.2, np.float32))
    return sc


CAM = dr.camera(dr.LENS_PINHOLE, position=(0.0, 0.0, -0.97), angle=60.0)


@pytest.mark.parametrize("level,blocks", [(0, 1), (0, 8), (0, 9), (3, 8), (3, 9)])   # 1,024 + n / 256 paths and 128 more
def test_calls_of_few_and_many_paths_agree(cuda, level, blocks):
    sc, r = _scene(level), dr.Renderer(1 << 14)
    params = dr.render_params(64, 64, dr.MODE_PHYSICAL, samples=(1, 1), max_bounces=3, seed=9)
    dl = dr.new_frame_buffer(64, 64, cuda)
    dl[:, :3] = torch.rand((len(dl), 3), generator=torch.Generator(cuda).manual_seed(1), device=cuda) + 0.1
    got = torch.rand((2, sc.n, 3), generator=torch.Generator(cuda).manual_seed(2), device=cuda)
    want = got.double()
    r.render_adjoint(sc, CAM, dl, 0, blocks, params, got[0], got[1])
    for b in range(blocks):
        part = torch.zeros_like(got)
        r.render_adjoint(sc, CAM, dl, b, b + 1, params, part[0], part[1])
        want += part.double()
    assert torch.allclose(got.double(), want, rtol=6e-4, atol=6e-8)


def test_a_captured_call_holds_when_a_larger_scene_comes(cuda):
    small, large, r = _scene(0), _scene(4), dr.Renderer(1 << 14)
    params = dr.render_params(64, 64, dr.MODE_PHYSICAL, samples=(1, 1), max_bounces=3, seed=9)
    nb = dr.block_count(64, 64)
    dl = dr.new_frame_buffer(64, 64, cuda) + 0.5
    one, got, other = (torch.zeros((2, s.n, 3), device=cuda) for s in (small, small, large))
    r.render_adjoint(small, CAM, dl, 0, nb, params, one[0], one[1])   # allocates what the capture may not
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        r.render_adjoint(small, CAM, dl, 0, nb, params, got[0], got[1])
    for _ in range(2):
        r.render_adjoint(large, CAM, dl, 0, nb, params, other[0], other[1])
        graph.replay()
    torch.cuda.synchronize()
    assert torch.allclose(got.double(), 2 * one.double(), rtol=1.2e-3, atol=1e-7)
    assert (other > 0).any()
