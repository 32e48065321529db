"""closestPointToPoint, four lanes per query, on both sides of the line where it takes over from whole warps, with
queries that are still walked when a warp has nothing else left and go to all its lanes: points about as far from
every triangle of a sphere, among them its centre, where nearly all candidates are undecided."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(pkg, name):
    if name == "sphere":
        return pkg.sphere(10.0, 48, 32), {}
    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    if name == "leaf":
        g.index = g.index[:120]
        return g, {"maxLeafSize": 64}
    if name == "groups":
        g.add_group(0, 900, 0)
        g.add_group(1200, 1500, 1)
        g.add_group(3000, 600, 2)
    return g, {}


@pytest.mark.parametrize("mesh", ["sphere", "leaf", "groups"])
@pytest.mark.parametrize("n", [32768, 32769, 40_003, 151_553])
@pytest.mark.parametrize("far", [math.inf, 9.9])
def test_handed_over_queries(pkg, cuda, mesh, n, far):
    import torch

    g, opts = _mesh(pkg, mesh)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, **opts})
    rng = np.random.default_rng(n)
    c = 0.5 * (g.position.min(0) + g.position.max(0))
    pts = (c + rng.normal(0, 5, (n, 3))).astype(np.float32)
    pts[::97] = c + rng.normal(0, 1e-3, (len(pts[::97]), 3))      # one in three warps' chunks has such a point
    pts[::1009] = c
    pts[5::2003] = np.nan
    d = torch.from_numpy(pts.astype(np.float32)).to(cuda)
    bvh.set_traversal(closest=0)
    want = bvh.closest_point_batch(d, 1e-30, far)
    got = bvh.closest_point_batch(d, 0.0, far)
    bvh.synchronize()
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
