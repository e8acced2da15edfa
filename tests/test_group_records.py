"""The 256-byte group records that a cast descends by.

A record finds a child without reading its node, which needs the inner children's groups and the leaf
children's references to be consecutive (checked on exported trees of both paddings and several
shapes), and it tests the children's boxes with a fused, widened slab test, which must never lose a
leaf: casts whose directions have zero, negative-zero and vanishing components, whose lengths are far
from 1 or whose origins lie on box planes or far outside equal the oracle's, index and t bit for bit."""
import numpy as np
import pytest

import dumbray_gb300 as dr
from dumbray_gb300 import scenes

SHAPES = {
    "mesh": lambda: np.concatenate([scenes.displaced_icosphere(4, 0.1, 2), scenes.box((3.0, 3.0, 3.0), inward=True)]),
    "boxes": lambda: scenes.random_boxes(400, np.random.default_rng(3)),
    "plane": lambda: scenes.quad((0.0, -1.4, 0.0), (6.0, 6.0), (0.0, 1.0, 0.0)),
    "corner": lambda: np.concatenate([scenes.icosphere(2, 1e-3, (5.0, 5.0, 5.0)), scenes.box((20.0, 20.0, 20.0))]),
    "offset": lambda: scenes.displaced_icosphere(3, 0.1, 1, center=(300.0, -40.0, 7.0)),
}


@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("split,eps", [(0, 0.0), (2, dr.PHYSICAL_TREE), (8, dr.PHYSICAL_TREE)])
def test_siblings_are_consecutive(shape, split, eps):
    _, _, child, leaf, _ = dr.build_octree_host(SHAPES[shape](), split_threshold=split, box_epsilon=eps)
    for g in range(1, len(child), 8):
        c, l = child[g:g + 8], leaf[g:g + 8]
        inner = c[c >= 0]
        assert np.array_equal(inner, inner[:1].repeat(len(inner)) + 8 * np.arange(len(inner)))
        l = l[c < 0]
        assert np.array_equal(l[1:, 0], (l[:-1, 0] + l[:-1, 1]))


def _rays(tris, box):
    rng = np.random.default_rng(11)
    lo, hi = tris.reshape(-1, 3).min(0), tris.reshape(-1, 3).max(0)
    size = (hi - lo).max()
    o, d = scenes.incoherent_rays(6000, lo - 0.2 * size, hi + 0.2 * size, seed=5)
    k = np.arange(len(o))
    for axis in range(3):                       # one or two components zero, -0 or vanishing
        d[k % 11 == axis, axis] = 0.0
        d[k % 13 == axis, axis] = -0.0
        d[k % 17 == axis, axis] *= np.float32(1e-13)
        d[k % 19 == axis, (axis + 1) % 3] = 0.0
        d[k % 19 == axis, (axis + 2) % 3] = 0.0
    planes = box[rng.integers(0, len(box), len(o))]
    for axis in range(3):                       # origins on the planes of node boxes
        at = k % 7 == axis
        o[at, axis] = np.where(rng.random(at.sum()) < 0.5, planes[at, axis], planes[at, 3 + axis])
    far = k % 23 == 0
    o[far] -= d[far] * np.float32(40.0) * size
    for i, s in enumerate((1e-15, 1e-6, 1e6, 1e15)):
        d[k % 29 == i] *= np.float32(s)
    d[k % 31 == 0] = 0.0
    d[k % 211 == 1, 1] = np.nan
    d[k % 223 == 2, 2] = np.inf
    o[k % 227 == 3, 0] = np.inf
    o[k % 229 == 4] *= np.float32(1e30)
    return o, d


@pytest.mark.gpu
@pytest.mark.parametrize("shape", sorted(SHAPES))
@pytest.mark.parametrize("cull", [True, False])
def test_casts_equal_the_oracle_on_awkward_rays(cuda, shape, cull):
    import torch

    import _oracle as O
    tris = SHAPES[shape]()
    sc = dr.Scene(tris)
    o, d = _rays(tris, sc.export_tree()[0])
    tri, t = dr.cast(sc, torch.from_numpy(o).to(cuda), torch.from_numpy(d).to(cuda), cull_backfaces=cull)
    tri, t = tri.cpu().numpy(), t.cpu().numpy()
    oi, ot, _, _ = O.OracleScene(tris).cast(o, d, cull=cull)
    assert np.array_equal(tri, oi), f"{(tri != oi).sum()} index mismatches"
    hit = oi >= 0
    assert np.array_equal(t[hit].view(np.int32), ot[hit].view(np.int32))
