"""Exactly equal hits: rays through vertices that several triangles share.  One ray per thread in the reference's
order of visits finds the triangle that the reference finds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sx,sy", [(1, 1), (-1, 1), (1, -1), (-1, -1)])
@pytest.mark.parametrize("leaf", [1, 4, 10])
def test_the_reference_order_keeps_the_first(pkg, orc, cuda, sx, sy, leaf):
    import torch

    k = 33                                   # a plane of unit squares, and rays whose every number is exact
    i = np.arange(k - 1)[:, None] * k + np.arange(k - 1)[None]
    index = np.stack([i, i + 1, i + k, i + 1, i + k + 1, i + k], -1).reshape(-1).astype(np.uint32)
    x, y = np.meshgrid(np.arange(k, dtype=np.float32), np.arange(k, dtype=np.float32))
    g = pkg.Geometry(np.stack([x, y, 0 * x], -1).reshape(-1, 3), index)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, "maxLeafSize": leaf})
    ref = orc.OracleBVH.from_serialized(bvh._roots, g.index, bvh._indirectBuffer, g.position)
    at = g.position[(x > 0).reshape(-1) & (y > 0).reshape(-1) & (x < k - 1).reshape(-1) & (y < k - 1).reshape(-1)]
    d = np.array([sx * 0.5, sy * 0.25, -1.0], np.float32)
    rays = np.concatenate([at - 8 * d, np.broadcast_to(d, at.shape)], 1).astype(np.float32)
    want = ref.raycast_first(rays, 2)
    bvh.set_traversal(0, 0)
    got = bvh.raycast_first_batch(torch.from_numpy(rays).to(cuda), 2)
    bvh.synchronize()
    assert np.array_equal(got.cpu().numpy().view(np.uint32)[:, 0].astype(np.int64), want["face_index"])
