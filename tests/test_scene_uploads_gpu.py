"""Scene arrays that go up in one copy and those that go up one by one make the same scene.

Host-built scenes upload the tree and are staged below 1 MiB; device-built ones have the tree on the device
already; the material ids alone pass 1 MiB from 262,144 triangles on.  Both builds are the same tree, so casts
agree to the bit and a frame, which reads the normals, materials and lights too, up to the order of its sums."""
import numpy as np
import pytest
import torch

import dumbray_gb300 as dr
from dumbray_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("normals", [False, True])
@pytest.mark.parametrize("n", [1, 2, 9, 1280, 5000, 9000, 262100, 262200])
def test_host_and_device_built_scenes_agree(cuda, n, normals):
    tris = scenes.icosphere(7 if n > 20480 else 5)[:n]
    rng = np.random.default_rng(n)
    nrm = (tris + rng.normal(0, 0.1, tris.shape)).astype(np.float32) if normals else None
    mats = [dr.dumb_based(diffuse=(0.7, 0.5, 0.3), metal=0.2), dr.simple_stochastic((0.9, 0.8, 0.7), 0.6, 0.4, 8.0)]
    lights = [dr.spherical_light((3.0, 3.0, 3.0), (0.0, 2.5, -2.0), 0.1), dr.directional_light((0.5, 0.5, 0.5), (0.0, -1.0, 1.0), 10.0)]
    mat = rng.integers(0, 2, n).astype(np.int32)
    scene = [dr.Scene(tris, normals=nrm, mat_id=mat, materials=mats, lights=lights, device_build=b) for b in (False, True)]
    at = tris[rng.integers(0, n, 4000)].mean(1)
    o = (at * 2.0 + rng.normal(0, 0.3, at.shape)).astype(np.float32)
    o, d = torch.from_numpy(o).to(cuda), torch.from_numpy((at - o).astype(np.float32)).to(cuda)
    host, device = (dr.cast(s, o, d, cull_backfaces=False) for s in scene)
    assert torch.equal(host[0], device[0]) and torch.equal(host[1], device[1])
    assert (host[0] >= 0).any()
    cam = dr.camera(dr.LENS_SIMPLE_STOCHASTIC, position=tuple(float(x) for x in 2.5 * tris[0].mean(0)), target=tuple(float(x) for x in tris[0].mean(0)))
    params = dr.render_params(40, 24, dr.MODE_REFERENCE, samples=(1, 1), max_bounces=2, cull_backfaces=False, seed=4)
    frames = []
    for s in scene:
        fb = dr.new_frame_buffer(40, 24, cuda)
        dr.Renderer(1 << 12).render_blocks(s, cam, fb, 0, dr.block_count(40, 24), params)
        torch.cuda.synchronize()
        frames.append(fb)
    assert torch.allclose(*frames, rtol=1e-5, atol=1e-6)
    assert n < 1280 or (frames[0][:, :3] > 0).any()   # fewer are smaller than a pixel
