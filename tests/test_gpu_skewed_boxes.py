"""intersectsBox with boxes whose edges are not at right angles, or flat: the reference's axes do not separate all
that is apart then, and a triangle counts as met although its part of the leaf, or its own bounds, lie apart."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _boxes(g, n, kind, seed):
    rng = np.random.default_rng(seed)
    q, _ = np.linalg.qr(rng.standard_normal((n, 3, 3)))
    p, _ = np.linalg.qr(rng.standard_normal((n, 3, 3)))
    scale = np.exp(rng.uniform(-3, 1, (n, 3)))
    a = q * scale[:, None, :]
    if kind == "sheared":
        a = a @ p
    elif kind == "flat":                       # one edge, or two, of length zero
        a[np.arange(n), :, rng.integers(0, 3, n)] = 0
        a[::5, :, 0] = 0
    elif kind == "nearly right":
        a = a + rng.normal(0, 1e-6, a.shape)
    b = np.zeros((n, 24), np.float32)
    half = rng.random((n, 3)) + 0.05
    b[:, 0:3], b[:, 4:7] = -half, half
    for k in range(3):
        b[:, 8 + 4 * k:11 + 4 * k] = a[:, :, k]
    lo, hi = g.position.min(0) - 1, g.position.max(0) + 1
    b[:, 20:23] = lo + rng.random((n, 3)) * (hi - lo)
    b[:, 23] = 1
    return b


@pytest.mark.parametrize("kind", ["right", "nearly right", "sheared", "flat"])
@pytest.mark.parametrize("leaf", [10, 40, 2000])
@pytest.mark.parametrize("n", [3000, 30_000, 40_000])
def test_against_the_oracle(pkg, orc, cuda, kind, leaf, n):
    import torch

    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH, "maxLeafSize": leaf})
    ref = orc.OracleBVH.from_serialized(bvh._roots, g.index, bvh._indirectBuffer, g.position)
    b = _boxes(g, n, kind, n + leaf)
    want = ref.intersects_box(b)
    got = bvh.intersects_box_batch(torch.from_numpy(b).to(cuda))
    bvh.synchronize()
    assert 0.02 < want.mean() < 0.98
    assert np.array_equal(got.cpu().numpy().astype(bool), want)
