"""near and far that are not numbers, negative, infinite or swapped: every form of the raycasts answers as one thread
per ray over child pairs does.  No node box passes a near that is not a number, but a root that is a leaf has no
box to test."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
NAN, INF = math.nan, math.inf


def _mesh(pkg, name):
    if name == "triangle":
        return pkg.Geometry(np.array([[0, 0, 0], [4, 0, 0], [0, 4, 0]], np.float32), np.array([0, 1, 2], np.uint16)), {}
    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    if name == "leaf40":
        g.index = g.index[:120]
    return g, {"maxLeafSize": 64} if name == "leaf40" else {}


def _rays(pkg, n):
    r = pkg.rays_sphere_to_box(n, seed=n)
    r[1::2, :3] *= np.float32(0.3)
    return r


@pytest.mark.parametrize("mesh", ["triangle", "leaf40", "plain"])
@pytest.mark.parametrize("near,far", [(NAN, INF), (0.0, NAN), (NAN, NAN), (-1.0, INF), (0.0, -1.0), (INF, INF),
                                      (30.0, 10.0), (-INF, INF), (2.0, 35.0)])
def test_first_hits(pkg, cuda, mesh, near, far):
    import torch

    g, opts = _mesh(pkg, mesh)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, **opts})
    for n in (500, 30_000, 200_000):
        rays = torch.from_numpy(_rays(pkg, n)).to(cuda)
        for leaf in (0, 4):
            bvh.set_leaf_size(leaf)
            bvh.set_traversal(0, 1)
            want = bvh.raycast_first_batch(rays, 2, near, far)
            for kw in (dict(persistent=1), dict(persistent=2), dict(persistent=2, wide=1)):
                bvh.set_traversal(**kw)
                got = bvh.raycast_first_batch(rays, 2, near, far)
                bvh.synchronize()
                assert torch.equal(got.view(torch.int32), want.view(torch.int32)), (n, leaf, kw)


@pytest.mark.parametrize("mesh", ["triangle", "leaf40", "plain"])
@pytest.mark.parametrize("near,far", [(NAN, INF), (0.0, NAN), (NAN, NAN), (0.0, -1.0), (30.0, 10.0), (2.0, 35.0)])
def test_all_hits(pkg, cuda, mesh, near, far):
    import torch

    g, opts = _mesh(pkg, mesh)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, **opts})
    rays = torch.from_numpy(_rays(pkg, 20_000)).to(cuda)
    bvh.set_traversal(all=0)
    want = bvh.raycast_batch(rays, 2, near, far, cap=4)[0]
    bvh.set_traversal(all=1)
    got = bvh.raycast_batch(rays, 2, near, far, cap=4)[0]
    bvh.synchronize()
    assert torch.equal(got, want)
