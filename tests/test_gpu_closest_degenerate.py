"""closestPointToPoint on meshes with triangles two of whose corners coincide: with the first two, the closest
point on their first edge is 0 / 0 where that edge is the nearest region, in the reference's arithmetic too, which
then does not take them; with the last two they are segments.  Every form against the oracle, whatever lane meets them first."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mesh(pkg, only):
    """A knot with a quarter of its triangles (the lowest face indices among them) degenerate: a = b, b = c,
    a = c, or all three; or nothing but a = b."""
    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    tri = g.index.reshape(-1, 3).copy()
    k = np.arange(len(tri))
    pick = np.ones(len(tri), bool) if only else (k < 40) | (k % 5 == 0)
    kind = np.zeros(len(tri), int) if only else np.where(k % 2 == 0, 0, 1 + k % 7 % 3)
    for which, (to, of) in enumerate(((1, 0), (2, 1), (2, 0))):
        rows = pick & (kind == which)
        tri[rows, to] = tri[rows, of]
    tri[pick & (kind == 3)] = tri[pick & (kind == 3)][:, :1]
    g.index = tri.reshape(-1).astype(g.index.dtype)
    return g


@pytest.mark.parametrize("only", [False, True])
@pytest.mark.parametrize("leaf", [1, 10, 2000])
@pytest.mark.parametrize("n", [33, 4097, 200_001])
def test_degenerate_triangles(pkg, orc, cuda, only, leaf, n):
    import torch

    g = _mesh(pkg, only)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, "maxLeafSize": leaf})
    ref = orc.OracleBVH.from_serialized(bvh._roots, g.index, bvh._indirectBuffer, g.position)
    rng = np.random.default_rng(n)
    v = g.position[g.index.reshape(-1, 3)]
    pts = (v[rng.integers(0, len(v), n), rng.integers(0, 3, n)] + rng.normal(0, 0.5, (n, 3))).astype(np.float32)
    pts[::3] = v[rng.integers(0, len(v), len(pts[::3])), 0]                 # on a corner
    pts[1::3] = (0.5 * (v[:, 0] + v[:, 2]))[rng.integers(0, len(v), len(pts[1::3]))]  # on the degenerate edge
    check = np.arange(n) if n < 5000 else rng.integers(0, n, 4000)
    want = ref.closest_point(pts[check])
    d = torch.from_numpy(pts).to(cuda)
    first = None
    for kw in (dict(closest=0), dict(closest=1), dict(closest=1, tile=32, tile_rows=4), dict(closest=2)):
        for low in (0.0, 1e-30):               # the per-query kernel too
            bvh.set_traversal(**kw)
            got = bvh.closest_point_batch(d, low, math.inf)
            bvh.synchronize()
            got = got.cpu().numpy()
            assert not np.isnan(got[:, 1:]).any(), kw
            if low == 0.0:
                first = got if first is None else first
                assert np.array_equal(first.view(np.int32), got.view(np.int32)), kw
            face, dist = got.view(np.uint32)[check, 0], got[check, 1]
            none = want["face_index"] < 0
            assert np.array_equal(face == 0xFFFFFFFF, none), kw
            assert (np.abs(dist - want["distance"])[~none] <= 1e-5 * np.maximum(want["distance"], 1e-3)[~none]).all(), kw
