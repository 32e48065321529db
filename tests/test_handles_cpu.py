"""The handle code (csrc/api.cu) over a stand-in for the CUDA runtime: what a call leaves behind when an
allocation in it fails."""
import ctypes as C
import importlib
import os
import subprocess

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
OK, OOM = 0, 4


@pytest.fixture(scope="module")
def lib(pkg, tmp_path_factory):
    out = tmp_path_factory.mktemp("fake") / "libfake.so"
    csrc = os.path.join(ROOT, "three-mesh-bvh_b200", "csrc")
    cuda = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include")
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic", "-include", "cmath",
                    "-I", csrc, "-I", os.path.join(ROOT, "include"), "-I", cuda, "-x", "c++", os.path.join(csrc, "api.cu"),
                    os.path.join(csrc, "builder.cpp"), os.path.join(ROOT, "tests", "native", "fake_cuda.cpp"),
                    "-o", str(out)], check=True)
    # lazily bound (ctypes itself binds at once): the launches that no test reaches are not there
    dlopen = C.CDLL(None).dlopen
    dlopen.restype, dlopen.argtypes = C.c_void_p, [C.c_char_p, C.c_int]
    dll = C.CDLL(str(out), handle=dlopen(str(out).encode(), os.RTLD_LAZY))
    native = importlib.import_module(pkg.__name__ + "._native")
    for name, res, args in native.SIGNATURES:
        if hasattr(dll, name):
            getattr(dll, name).restype, getattr(dll, name).argtypes = res, args
    dll.fake_held.restype = C.c_int64
    return dll


def _mesh(pkg, lib):
    g = pkg.torus_knot(10, 3, 60, 12, noise_sigma=0.05, noise_seed=3)
    bvh = pkg.MeshBVH(g, {"strategy": pkg.SAH})
    bufs = [np.frombuffer(r, np.uint8) for r in bvh._roots]
    ptrs, sizes = (C.c_void_p * 1)(bufs[0].ctypes.data), (C.c_uint64 * 1)(bufs[0].size)
    pos, out = np.ascontiguousarray(g.position, np.float32), C.c_void_p()
    args = (0, 1, ptrs, sizes, 1, g.index.ctypes.data, g.index.dtype.itemsize, g.index.size, None, 0, 0,
            pos.ctypes.data, pos.shape[0], 3)
    return args, out, (bvh, bufs, pos)


def test_a_leaf_layout_that_cannot_be_made_changes_nothing(pkg, lib):
    native = importlib.import_module(pkg.__name__ + "._native")
    args, mesh, keep = _mesh(pkg, lib)
    pos = keep[2]
    start = lib.fake_held()
    assert lib.bvhc_mesh_create(*args, C.byref(mesh)) == OK
    cfg = native.BvhcTraversalConfig(2, 0, 16, 2)
    assert lib.bvhc_mesh_set_traversal(mesh, C.byref(cfg)) == OK
    rays, hits = np.zeros((4, 6), np.float32), np.zeros((5, 8), np.float32)
    at = hits.ctypes.data + (-hits.ctypes.data) % 16

    def cast():
        before = lib.fake_packets()
        assert lib.bvhc_raycast_first(mesh, rays.ctypes.data, 4, 0, 0.0, 1e9, at, native.MEM_DEVICE, None) == OK
        assert lib.bvhc_mesh_refit(mesh, pos.ctypes.data, pos.shape[0], 3, native.MEM_DEVICE, None) == OK
        assert lib.fake_packets() == before + 1 and lib.fake_bad() == 0

    cast()
    for old, new in ((0, 3), (3, 1), (1, 2)):
        failures = 0
        while True:
            held = lib.fake_held()
            lib.fake_fail_in(failures + 1)
            status = lib.bvhc_mesh_set_leaf_size(mesh, new)
            if lib.fake_fail_left() > 0:        # every allocation of the call was made
                lib.fake_fail_in(0)
                break
            assert status == OOM
            assert lib.bvhc_mesh_get_leaf_size(mesh) == old and lib.fake_held() == held
            cast()
            failures += 1
        assert status == OK and failures > 8 and lib.bvhc_mesh_get_leaf_size(mesh) == new
        cast()
    assert lib.bvhc_mesh_set_leaf_size(mesh, 0) == OK
    cast()
    lib.bvhc_mesh_destroy(mesh)
    assert lib.fake_held() == start and lib.fake_bad() == 0


def test_handles_made_for_one_pick_share_page_locked_memory(pkg, lib):
    native = importlib.import_module(pkg.__name__ + "._native")
    args, _, keep = _mesh(pkg, lib)
    rays, hits = np.zeros((4, 6), np.float32), np.zeros((4, 8), np.float32)
    cfg = native.BvhcTraversalConfig(2, 0, 16, 2)

    def pick():
        mesh = C.c_void_p()
        assert lib.bvhc_mesh_create(*args, C.byref(mesh)) == OK
        assert lib.bvhc_mesh_set_traversal(mesh, C.byref(cfg)) == OK
        assert lib.bvhc_raycast_first(mesh, rays.ctypes.data, 4, 0, 0.0, 1e9, hits.ctypes.data, native.MEM_HOST, None) == OK
        return mesh

    before, held = lib.fake_host_blocks(), lib.fake_held()
    for _ in range(5):
        lib.bvhc_mesh_destroy(pick())
    assert lib.fake_host_blocks() == before + 1
    meshes = [pick() for _ in range(7)]                      # one block each while they live
    assert lib.fake_host_blocks() == before + 7
    for mesh in meshes:
        lib.bvhc_mesh_destroy(mesh)
    assert lib.fake_held() == held + 4                       # no more are kept than four
    lib.fake_lose_host(1)                                    # nor used once their context is gone
    mesh = pick()
    lib.fake_lose_host(0)
    lib.bvhc_mesh_destroy(mesh)
    assert lib.fake_host_blocks() == before + 8 and lib.fake_bad() == 0
