"""Casts along an axis from far away: the group tests keep every box that the exact slab test keeps.

A direction component far below the largest is raised before the group test divides by it, which moves the
ray sideways by an amount that grows with the distance.  The floors lie at coordinate 0, so the distance of
the hit is the origin's to the bit, and the counting cast (exact slab tests) and the oracle find every one."""
import numpy as np
import pytest

import dumbray_gb300 as dr

pytestmark = pytest.mark.gpu
EXPONENTS = range(18, 42)
RAYS = 200      # a direction and an exponent


def _floor(axis, cells=32):
    """A square of side 1 at coordinate 0 of `axis`, two triangles a cell."""
    u = np.linspace(-0.5, 0.5, cells + 1, dtype=np.float32)
    a, b = np.meshgrid(u[:-1], u[:-1])
    s = np.float32(1.0 / cells)
    corner = lambda x, y: np.insert(np.stack([x.ravel(), y.ravel()], 1), axis, 0.0, 1)
    p, q, r, t = corner(a, b), corner(a + s, b), corner(a + s, b + s), corner(a, b + s)
    return np.concatenate([np.stack([p, q, r], 1), np.stack([p, r, t], 1)]).astype(np.float32)


def _rays(axis):
    rng = np.random.default_rng(axis)
    o, d = [], []
    for k in EXPONENTS:
        for side in (-1.0, 1.0):
            for small in (0.0, -0.0, 2.0 ** -100, -(2.0 ** -100)):   # the other components
                for length in (1.0, 1e-12, 1e12):
                    p = rng.uniform(-0.49, 0.49, (RAYS, 3)).astype(np.float32)
                    p[:, axis] = side * 2.0 ** k
                    v = np.full((RAYS, 3), small)
                    v[:, axis] = -side
                    o.append(p)
                    d.append((v * length).astype(np.float32))
    return np.concatenate(o), np.concatenate(d)


@pytest.mark.parametrize("axis", [0, 1, 2])
@pytest.mark.parametrize("split,eps", [(0, 0.0), (2, 0.0), (4, dr.PHYSICAL_TREE), (2, dr.PHYSICAL_TREE)])
def test_axis_parallel_rays_hit_from_any_distance(cuda, axis, split, eps):
    import torch

    import _oracle as O
    tris = _floor(axis)
    sc = dr.Scene(tris, split_threshold=split, box_epsilon=eps)
    o, d = _rays(axis)
    args = [torch.from_numpy(x).to(cuda) for x in (o, d)]
    tri, t = (x.cpu().numpy() for x in dr.cast(sc, *args, cull_backfaces=False))
    exact_tri, exact_t = (x.cpu().numpy() for x in dr.cast(sc, *args, cull_backfaces=False, counted=True)[:2])
    assert (exact_tri >= 0).all()
    lost = np.unique(np.abs(o[tri < 0, axis]))
    assert not len(lost), f"{(tri < 0).sum()} of {len(tri)} hits lost, from distances {lost}"
    assert np.array_equal(tri, exact_tri) and np.array_equal(t.view(np.int32), exact_t.view(np.int32))
    if eps == 0.0:
        oi, ot, _, _ = O.OracleScene(tris).cast(o, d, cull=False)
        assert np.array_equal(tri, oi) and np.array_equal(t.view(np.int32), ot.view(np.int32))
