"""Hits at distance 0 of either sign: the closest hit is the first in the list among equal distances, and -0 equals 0.

A ray that starts on a triangle's plane hits it when the product of direction and normal overflows (0 * inf is
not <= 0), at 0 or -0 by the signs.  Stacks of coplanar triangles that face either way, and slanted ones through
the same points with small distances, must give the oracle's triangle and distance to the bit."""
import numpy as np
import pytest
import torch

import dumbray_gb300 as dr
import _oracle as O

pytestmark = pytest.mark.gpu


def _tris(rng, count, flat):
    size = np.float32(3e4)
    t = rng.uniform(-1.0, 1.0, (count, 3, 3)).astype(np.float32) * size
    t[: int(flat * count), :, 1] = 0.0
    return t


@pytest.mark.parametrize("cull", [False, True])
@pytest.mark.parametrize("count,flat", [(3, 1.0), (40, 1.0), (40, 0.7), (400, 0.5)])
def test_ties_at_zero_go_to_the_first(cuda, count, flat, cull):
    rng = np.random.default_rng(count)
    tris = _tris(rng, count, flat)
    n = 20000
    o = rng.uniform(-2e4, 2e4, (n, 3)).astype(np.float32)
    o[:, 1] = np.where(np.arange(n) % 3 == 0, -0.0, 0.0)
    d = (rng.normal(0.0, 1.0, (n, 3)) * 10.0 ** rng.uniform(28.0, 34.0, (n, 1))).astype(np.float32)
    tri, t = (x.cpu().numpy() for x in dr.cast(dr.Scene(tris), torch.from_numpy(o).to(cuda), torch.from_numpy(d).to(cuda), cull_backfaces=cull))
    oi, ot, _, _ = O.OracleScene(tris).cast(o, d, cull=cull)
    hit = oi >= 0
    assert (np.signbit(ot[hit]) & (ot[hit] == 0.0)).any()
    assert np.array_equal(tri, oi), f"{(tri != oi).sum()} index mismatches"
    assert np.array_equal(t[hit].view(np.int32), ot[hit].view(np.int32))
