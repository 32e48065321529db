"""A leaf layout asked for after a refit holds the moved triangles."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_layout_after_refit(pkg, cuda):
    import torch

    g = pkg.torus_knot(10, 3, 80, 12, noise_sigma=0.05, noise_seed=4)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH})
    rays = torch.from_numpy(pkg.rays_sphere_to_box(20_000, seed=3)).to(cuda)
    before = bvh.raycast_first_batch(rays, 2)
    bvh.refit((g.position * 0.8 + 0.5).astype(np.float32))
    want = bvh.raycast_first_batch(rays, 2)
    assert not torch.equal(want[:, 1], before[:, 1])
    for leaf in (3, 1, 0, 2):
        bvh.set_leaf_size(leaf)
        for kw in (dict(persistent=1), dict(persistent=2)):
            bvh.set_traversal(**kw)
            got = bvh.raycast_first_batch(rays, 2)
            bvh.synchronize()
            assert torch.equal(got[:, 1], want[:, 1]), (leaf, kw)
