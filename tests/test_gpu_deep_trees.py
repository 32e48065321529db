"""A tree as deep as the traversal stacks allow whose last leaf is large: its four-child records, with the
leaf's parts, can stack more than the warp-shared form over them holds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chain", [50, 54, 55, 56, 57, 58, 59])
def test_every_form_fits_its_stack(pkg, cuda, chain):
    import torch

    # triangles across x at 1, 1/4, 1/16, ... (each split takes one off) and 64 more at x = 0
    x = np.concatenate([4.0 ** -np.arange(chain), np.zeros(64)])
    v = np.zeros((len(x), 3, 3), np.float32)
    v[:, :, 0] = x[:, None]
    v[:, :, 1], v[:, :, 2] = [-1, 1, 0], [-1, -1, 1]
    g = pkg.Geometry(v.reshape(-1, 3), np.arange(3 * len(x), dtype=np.uint32))
    bvh = pkg.MeshBVH(g, {"strategy": pkg.CENTER, "maxLeafSize": 64, "maxDepth": 100})
    assert bvh.mesh_info()["max_depth"] >= chain - 2
    n = 4096
    rays = np.zeros((n, 6), np.float32)
    rays[:, 0], rays[:, 3] = -1, 1
    rays[:, 1] = np.linspace(-0.9, 0.9, n)
    rays[n // 2:, 0], rays[n // 2:, 3] = 2, -1
    d = torch.from_numpy(rays).to(cuda)
    for leaf in (0, 8):
        bvh.set_leaf_size(leaf)
        bvh.set_traversal(0, 1)
        want = bvh.raycast_first_batch(d, 2)
        bvh.synchronize()
        assert (want.view(torch.int32)[:, 0] != -1).any()
        for kw in (dict(persistent=2, wide=1), dict(persistent=2, wide=0), dict(persistent=1)):
            bvh.set_traversal(**kw)
            got = bvh.raycast_first_batch(d, 2)
            bvh.synchronize()              # raises on a traversal stack overflow
            assert torch.equal(got[:, 1], want[:, 1]), (leaf, kw)
