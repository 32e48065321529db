"""raycastFirst at the batch sizes where one kernel takes over from another, four lanes per ray from whole warps and
one lane from four lanes, byte for byte against one thread per ray."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", ["leaf40", "leaves40", "groups"])
@pytest.mark.parametrize("n", [24576, 24577, 37_889, 196_608, 196_609, 230_001])
def test_both_sides_of_each_line(pkg, cuda, mesh, n):
    import torch

    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    opts = {}
    if mesh == "leaf40":
        g.index, opts = g.index[:120], {"maxLeafSize": 64}
    elif mesh == "leaves40":
        opts = {"maxLeafSize": 40}
    else:
        for start, count, k in ((0, 900, 0), (1200, 1500, 1), (3000, 600, 2)):
            g.add_group(start, count, k)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, **opts})
    r = np.concatenate([pkg.rays_sphere_to_box(n, seed=n), pkg.rays_incoherent(n, seed=n + 1)])[n // 2:n // 2 + n]
    r[::5, 3:] *= np.float32(3.5)
    r[1::7, 3] = 0.0
    rays = torch.from_numpy(r).to(cuda)
    for leaf in (0, 3):
        bvh.set_leaf_size(leaf)
        for compact, sort in ((0, 0), (1, 0), (1, 3)):
            for side, near, far in ((0, 0.0, math.inf), (1, 20.0, 45.0), (2, -5.0, 38.0)):
                bvh.set_traversal(0, 1)
                want = bvh.raycast_first_batch(rays, side, near, far)
                bvh.set_traversal(1, 1, 16, 0, compact, sort)
                got = bvh.raycast_first_batch(rays, side, near, far)
                bvh.synchronize()
                assert torch.equal(got.view(torch.int32), want.view(torch.int32)), (leaf, compact, sort, side)
