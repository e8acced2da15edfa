"""A batch whose ray coordinates number more than 2^31: the last rays are the last rays."""
import pytest
import torch

import dumbray_gb300 as dr
from dumbray_gb300 import scenes

pytestmark = pytest.mark.gpu


def test_rays_past_two_to_the_31_coordinates(cuda):
    n = (1 << 31) // 3 + 100003
    if torch.cuda.mem_get_info()[0] < 3 * 32 * n // 2:
        pytest.skip("needs 35 GB")
    sc = dr.Scene(scenes.quad((0.0, 0.0, 0.0), (2.0, 2.0), (0.0, 1.0, 0.0)))
    o, d = torch.empty((n, 3), device=cuda), torch.zeros((n, 3), device=cuda)
    o[:] = torch.tensor([5.0, 1.0, 0.0], device=cuda)      # beside the quad
    d[:, 1] = -1.0
    hits = torch.cat([torch.arange(0, n, 1_000_003, device=cuda), torch.arange(n - 70000, n, 7, device=cuda)]).unique()
    o[hits, 0] = 0.25
    o[hits, 1] = 1.0 + (hits % 1000) / 1024.0
    tri, t = dr.cast(sc, o, d)
    assert int((tri >= 0).sum()) == len(hits)
    assert torch.equal(t[hits], o[hits, 1])
