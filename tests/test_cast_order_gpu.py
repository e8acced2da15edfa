"""Large batches whose neighbours go the same way are cast in another order: every ray's result is the one it
has in a small batch, to the bit, whatever the order, the remainder and the counters."""
import numpy as np
import pytest
import torch

import dumbray_gb300 as dr
from dumbray_gb300 import scenes

pytestmark = pytest.mark.gpu
SMALL = 1 << 14      # far below a ray for every lane: rays in their order


@pytest.fixture(scope="module")
def scene(cuda):
    return dr.Scene(scenes.displaced_icosphere(5))


@pytest.mark.parametrize("counted", [False, True])
@pytest.mark.parametrize("extra", [-1, 0, 1, 31, 32, 45, "twice"])
@pytest.mark.parametrize("kind", ["coherent", "random", "half", "zero"])
def test_batches_equal_small_batches(cuda, scene, kind, extra, counted):
    lanes = torch.cuda.get_device_properties(0).multi_processor_count * (768 if counted else 1024)
    n = 2 * lanes + 77 if extra == "twice" else lanes + extra
    g = torch.Generator(cuda).manual_seed(n)
    k = torch.arange(n, device=cuda)
    side = 400
    d = torch.stack([(k % side) / side - 0.5, (k // side) / (n // side + 1) - 0.5, torch.ones_like(k)], 1).float()
    o = torch.tensor([0.0, 0.0, -2.6], device=cuda).repeat(n, 1)
    if kind == "random" or kind == "half":
        part = n if kind == "random" else n // 2
        d[:part] = torch.randn((part, 3), generator=g, device=cuda)
        o[:part] = -1.3 * d[:part] / d[:part].norm(dim=1, keepdim=True) + 0.5 * torch.randn((part, 3), generator=g, device=cuda)
    if kind == "zero":
        d[::3] = 0.0
        d[1::7] = float("nan")
    ignore = torch.randint(-1, scene.n, (n,), generator=g, device=cuda, dtype=torch.int32)
    got = dr.cast(scene, o, d, ignore=ignore, counted=counted)
    for a in range(0, n, SMALL):
        want = dr.cast(scene, o[a:a + SMALL].contiguous(), d[a:a + SMALL].contiguous(), ignore=ignore[a:a + SMALL].contiguous(), counted=counted)
        for x, y in zip(got, want):
            assert torch.equal(x[a:a + SMALL], y)
    assert (got[0] >= 0).any()
