"""raycastFirst over triangles whose corners are not numbers or infinite, with low face indices among them: their
determinants can leave a hit at a distance that is not a number, which may not keep or take the place of one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("leaf", [4, 10, 2000])
@pytest.mark.parametrize("what", [np.nan, np.inf, -np.inf])
def test_first_hits(pkg, orc, cuda, leaf, what):
    import torch

    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    bad = g.index.reshape(-1, 3)[::7].copy()          # every seventh triangle gets corners of its own
    first = g.position.shape[0]
    own = g.position[bad].copy()
    own[::2, 1] = what
    own[1::2, 2, 1] = what
    g.position = np.concatenate([g.position, own.reshape(-1, 3)]).astype(np.float32)
    index = g.index.reshape(-1, 3).copy()
    index[::7] = first + np.arange(3 * len(bad)).reshape(-1, 3)
    g.index = index.reshape(-1).astype(np.uint32)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.CENTER, "maxLeafSize": leaf})
    ref = orc.OracleBVH.from_serialized(bvh._roots, g.index, bvh._indirectBuffer, g.position)
    for n in (500, 30_000, 200_000):
        r = pkg.rays_sphere_to_box(n, seed=n)
        want = ref.raycast_first(r[:20_000], 2)
        d = torch.from_numpy(r).to(cuda)
        for kw in (dict(persistent=0, order=0), dict(persistent=0, order=1), dict(persistent=1), dict(persistent=2),
                   dict(persistent=2, wide=1)):
            bvh.set_traversal(**kw)
            got = bvh.raycast_first_batch(d, 2)
            bvh.synchronize()
            got = got.cpu().numpy()[:20_000]
            hit = got.view(np.uint32)[:, 0] != 0xFFFFFFFF
            assert not np.isnan(got[hit, 1]).any(), kw
            assert (hit == (want["face_index"] >= 0)).mean() == 1, kw
            assert (np.abs(got[hit, 1] - want["distance"][hit]) <= 1e-5 * want["distance"][hit]).all(), kw
