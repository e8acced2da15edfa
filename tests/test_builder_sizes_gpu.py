"""GPU octree build at the sizes where its passes change shape: staged sums of 128, reference lists of
2,048 (a warp up to that, the block beyond), block chunks of 1,024, scan chunks; against the host build,
bit for bit."""
import numpy as np
import pytest

import dumbray_gb300 as dr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [31, 32, 33, 127, 128, 129, 1023, 1025, 2047, 2048, 2049, 3071, 3073, 8191, 8193, 20001])
@pytest.mark.parametrize("eps", [0.0, dr.PHYSICAL_TREE])
def test_device_build_at_pass_sizes(cuda, n, eps):
    rng = np.random.default_rng(n)
    # mostly small triangles, some crossing many octants, a flat patch lying on one plane
    size = np.where(rng.random((n, 1, 1)) < 0.05, 0.5, 0.02)
    tris = (rng.uniform(-1.0, 1.0, (n, 1, 3)) + size * rng.normal(size=(n, 3, 3))).astype(np.float32)
    tris[: n // 8, :, 1] = 0.25
    a = dr.build_octree_host(tris, box_epsilon=eps)
    b = dr.build_octree_host(tris, box_epsilon=eps, device_build=True)
    assert a[0] == b[0]
    for x, y in zip(a[1:], b[1:]):
        assert np.array_equal(np.asarray(x).view(np.int32), np.asarray(y).view(np.int32))
