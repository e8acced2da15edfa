"""Reference photons that pass a blocker, through each place they may wait for their next cast.

A veil under the light whose shader lets photons through (front to the light, so it is not culled): photons
stopped by it are kept by the filter and carried to the end of the wave; past a full carry region (1/16 of the
photon records, at least 1,024) they wait in the bounce's kept list; in a wave whose photons all fit they are
carried unshaded.  Single renders and batches, with and without counters, equal the oracle per pixel."""
import numpy as np
import pytest
import torch

import dumbray_gb300 as dr
from dumbray_gb300 import scenes
import _oracle as O

pytestmark = pytest.mark.gpu
CARRY = 1024        # carry capacity of a renderer of at most 8,192 paths a wave


def _scene():
    tris = [scenes.box((2.0, 2.0, 2.0), inward=True), scenes.icosphere(2, 0.4, (0.0, -0.4, 0.2)), scenes.quad((0.0, 0.55, 0.0), (1.9, 1.9), (0.0, 1.0, 0.0))]
    mat = np.repeat(np.arange(3), [len(t) for t in tris]).astype(np.int32)
    mats = [dr.dumb_based(diffuse=(0.7, 0.6, 0.5), metal=0.0), dr.dumb_based(diffuse=(0.3, 0.5, 0.7), metal=0.3),
            dr.simple_stochastic((0.9, 0.8, 0.7), 0.6, 0.4, 8.0)]
    lights = [dr.spherical_light((2.0, 2.0, 2.0), (0.0, 0.8, 0.0), 0.05), dr.spherical_light((1.0, 1.0, 1.5), (0.3, 0.8, -0.3), 0.05)]
    args = dict(mat_id=mat, materials=mats, lights=lights)
    tris = np.concatenate(tris).astype(np.float32)
    return dr.Scene(tris, **args), O.OracleScene(tris, **args)


# resolution, samples and depth of a job (every job a wave of its own or part of one), jobs, paths a wave, what
# the photons that go on do
CASES = {
    "kept list": (16, 2, 4, 1, 1024, "overflow"),
    "kept list, batch": (16, 1, 4, 4, 1024, "overflow"),
    "carried": (16, 2, 4, 1, 1 << 16, "fit"),
    "unshaded": (16, 1, 2, 1, 1 << 14, "roomy"),
    "unshaded, batch": (8, 1, 2, 2, 1 << 14, "roomy"),
}


@pytest.mark.parametrize("counting", [True, False])
@pytest.mark.parametrize("case", sorted(CASES))
def test_photons_past_a_veil_equal_the_oracle(cuda, case, counting):
    side, s, depth, jobs, wave, way = CASES[case]
    sc, osc = _scene()
    cam = dr.camera(dr.LENS_SIMPLE_STOCHASTIC, position=(0.0, -0.2, -0.95), angle=60.0)
    params = [dr.render_params(side, side, dr.MODE_REFERENCE, samples=(s, s), max_bounces=depth, seed=21 + j) for j in range(jobs)]
    nb = dr.block_count(side, side)
    fbs = [dr.new_frame_buffer(side, side, cuda) for _ in params]
    r = dr.Renderer(wave, 1)
    r.set_counting(counting)
    if jobs == 1:
        r.render_blocks(sc, cam, fbs[0], 0, nb, params[0])
    else:
        dr.Batch([(sc, cam, p, fb, 0, nb) for p, fb in zip(params, fbs)]).render(r, use_graph=not counting)
    torch.cuda.synchronize()
    photons = sum(r.wave_counts(depth + 1)[1])
    most = jobs * nb * 128 * s * s * (depth + 1) * 2     # one wave
    carry = max(CARRY, 2 * wave // 16)
    assert (most <= carry) == (way == "roomy")
    if counting:
        # no photon goes on more than twice (the veil has one layer, the sphere passes nothing from its front)
        on = r.counters()["shadow_casts"] - photons
        assert on > (2 * CARRY if way == "overflow" else 0) and (way == "overflow" or on <= carry), (photons, on)
    for p, fb in zip(params, fbs):
        gpu = dr.blockmajor_to_image(fb, side, side)[..., :3].astype(np.float64)
        ora = dr.blockmajor_to_image(osc.render_blocks(cam, p), side, side)[..., :3].astype(np.float64)
        # paths may split where a transcendental rounds differently: the bounds of the other oracle comparisons
        bad = np.abs(gpu - ora) > 2e-3 * np.maximum(np.abs(ora), 0.01)
        assert bad.mean() <= 0.02, f"{bad.mean():.4f} of channels differ"
        assert abs(gpu.mean() - ora.mean()) <= 5e-3 * ora.mean()
