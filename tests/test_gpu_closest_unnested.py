"""closestPointToPoint on a tree from a file whose boxes do not lie in their parents': it has no four-child records,
and the warp-shared forms over child pairs take it all the same, as the per-query kernel does."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("far", [math.inf, 2.0])
@pytest.mark.parametrize("n", [33, 5000, 210_000])
def test_forms_agree(pkg, cuda, n, far):
    import torch

    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    data = pkg.MeshBVH.serialize(pkg.MeshBVH(g, {"strategy": pkg.SAH}))
    nodes = np.frombuffer(data["roots"][0], np.float32).reshape(-1, 8).copy()
    count = nodes.view(np.uint32)[:, 7]
    for k in range(1, 40):
        if count[k] >> 16 != 0xFFFF:          # an inner node
            nodes[k, 3:6] += np.float32(0.02 * k)
    data["roots"] = [nodes.tobytes()]
    bvh = pkg.MeshBVH.deserialize(data, g)
    rng = np.random.default_rng(n)
    lo, hi = g.position.min(0) - 2, g.position.max(0) + 2
    pts = torch.from_numpy((lo + rng.random((n, 3)) * (hi - lo)).astype(np.float32)).to(cuda)
    bvh.set_traversal(closest=0)
    want = bvh.closest_point_batch(pts, 1e-30, far).view(torch.int32)
    for kw in (dict(closest=0), dict(closest=1), dict(closest=1, tile=32, tile_rows=4), dict(closest=2),
               dict(closest=3), dict(closest=6)):
        bvh.set_traversal(**kw)
        got = bvh.closest_point_batch(pts, 0.0, far)
        bvh.synchronize()
        assert torch.equal(got.view(torch.int32), want), kw
