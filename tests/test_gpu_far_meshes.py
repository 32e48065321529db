"""Rays with zero direction components on meshes far from the origin, where 1 / d stands for a huge number
and |o| / d can overflow: every form of the raycasts against a mesh whose root is one leaf, which tests
every triangle and no box (the distances and counts; equal ones may lie on either triangle of an edge)."""
import importlib
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _knot(pkg, offset):
    """A knot a hundredth of the offset in size, with one root of plain leaves, or all in one leaf."""
    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    far = np.abs(offset).max()
    g.position = (g.position * np.float32(far / 1000.0) + np.asarray(offset, np.float32)).astype(np.float32)
    return g


def _rays(g, n, seed):
    """Rays through the mesh's box, one or two direction components zero (of either sign)."""
    rng = np.random.default_rng(seed)
    lo, hi = g.position.min(0).astype(np.float64), g.position.max(0).astype(np.float64)
    at = lo + rng.random((n, 3)) * (hi - lo)
    d = rng.standard_normal((n, 3))
    axis = rng.integers(0, 3, n)
    one = np.arange(n) % 3 != 0
    d[np.arange(n), axis] = np.where(one, np.where(rng.random(n) < 0.5, 0.0, -0.0), d[np.arange(n), axis])
    two = np.arange(n) % 3 == 1
    d[two, (axis[two] + 1) % 3] = 0.0
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return np.concatenate([at - d * (hi - lo).max() * 1.5, d], 1).astype(np.float32)


OFFSETS = [(3e8, -3e8, 0), (-4e8, 4e8, 4e8), (1e9, 1e9, -1e9), (0, 1e9, 0), (1e12, 0, -1e12)]


@pytest.mark.parametrize("offset", OFFSETS)
def test_first_and_all_hits(pkg, cuda, offset):
    import torch

    g = _knot(pkg, offset)
    every = pkg.MeshBVH(g, {"strategy": pkg.SAH, "maxLeafSize": 2000})
    every.set_traversal(0, 1)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH})
    for n in (1000, 30_000, 200_000):
        rays = torch.from_numpy(_rays(g, n, n)).to(cuda)
        want = every.raycast_first_batch(rays, 2)[:, 1]
        assert 0.05 < torch.isfinite(want).float().mean() < 1
        for leaf in (0, 3):
            bvh.set_leaf_size(leaf)
            for kw in (dict(persistent=1), dict(persistent=1, compact=1), dict(persistent=2, order=0),
                       dict(persistent=2, order=1), dict(persistent=2, wide=1)):
                bvh.set_traversal(**kw)
                got = bvh.raycast_first_batch(rays, 2)[:, 1]
                bvh.synchronize()
                assert torch.equal(got, want), (n, leaf, kw)
    rays = rays[:20_000].contiguous()
    counts = every.raycast_batch(rays, 2, cap=8)[0]
    for variant in (0, 1):
        bvh.set_traversal(all=variant)
        got = bvh.raycast_batch(rays, 2, cap=8)[0]
        bvh.synchronize()
        assert torch.equal(got, counts), variant


@pytest.mark.parametrize("offset", OFFSETS)
def test_instances(pkg, cuda, offset):
    import torch

    batched = importlib.import_module(pkg.__name__ + ".batched")
    g = _knot(pkg, offset)
    m = np.zeros((70, 16))
    m[:, 0] = m[:, 5] = m[:, 10] = m[:, 15] = 1
    m[1:, 14] = np.arange(1, 70) * 1e3 * np.abs(offset).max()
    scenes = [batched.BatchedMeshBVH([g], {"strategy": pkg.SAH, "maxLeafSize": s}).instances(np.zeros(70, np.uint32), m)
              for s in (2000, 10)]
    rays = torch.from_numpy(_rays(g, 300, 5)).to(cuda)
    hits, inst = scenes[1].raycast_first(rays, 2)
    torch.cuda.synchronize()
    assert (inst == 0).float().mean() > 0.05
    for i in range(0, 300, 30):            # fewer than 32 rays a call: one thread per ray
        h, k = scenes[0].raycast_first(rays[i:i + 30].clone(), 2)
        torch.cuda.synchronize()
        assert torch.equal(k, inst[i:i + 30])
        assert torch.equal(h[:, 1], hits[i:i + 30, 1])


@pytest.mark.parametrize("length", [3e-30, 1e-15, 1e15])
def test_directions_far_from_unit_length(pkg, cuda, length):
    """An origin and a direction whose quotient overflows though no component is zero."""
    import torch

    g = _knot(pkg, (4e8, -4e8, 4e8))
    every = pkg.MeshBVH(g, {"strategy": pkg.SAH, "maxLeafSize": 2000})
    every.set_traversal(0, 1)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH})
    r = _rays(g, 200_000, 7)
    rng = np.random.default_rng(8)
    r[:, 3:] = (r[:, 3:] + (rng.random((200_000, 3)) * 2 - 1) * 0.01) * length
    for n in (1000, 30_000, 200_000):
        rays = torch.from_numpy(r[:n].copy()).to(cuda)
        want = every.raycast_first_batch(rays, 2)[:, 1]
        bvh.set_traversal(0, 1)
        per_ray = bvh.raycast_first_batch(rays, 2)[:, 1]
        for kw in (dict(persistent=1), dict(persistent=2)):
            bvh.set_traversal(**kw)
            got = bvh.raycast_first_batch(rays, 2)[:, 1]
            bvh.synchronize()
            found = torch.isfinite(per_ray) & (per_ray == want)
            assert torch.equal(got[found], want[found]), (n, kw)
