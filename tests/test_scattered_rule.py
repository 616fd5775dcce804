"""Which lmesh meshes run packed (scattered_mesh, csrc/host_setup.cpp): the count
of sectors a gather against a direct count, and on which side of the line the
meshes lie that the GPU tests of the packed kernels use."""
import ctypes
import os

import numpy as np
import pytest

import lmesh
from conftest import PKG


def islands(n, seed=0):
    """n cubes that share no node, element e's corner k at node 8 e + k, all a
    little distorted: every gather of 32 elements touches 32 sectors, whatever
    the size, so meshes from 28 elements up run packed."""
    rng = np.random.default_rng(seed)
    one = lmesh.box(1)
    xyz = np.concatenate([one.xyz + (0.0 if e == 0 else np.array([2.0 * e, 0.0, 0.0]) +
                                     0.05 * rng.uniform(-1.0, 1.0, (8, 3))) for e in range(n)])
    nodelist = np.concatenate([one.nodelist + 8 * e for e in range(n)])
    links = np.repeat(np.arange(n)[:, None], 6, axis=1)  # each face its own element
    return lmesh.LMesh(xyz, nodelist, links, one.symm, one.free)


def shuffled(nx):
    rng = np.random.default_rng(nx)
    return lmesh.renumber(lmesh.box(nx), rng.permutation((nx + 1) ** 3), rng.permutation(nx ** 3))


def rule(tmp_path, mesh):
    """(sectors a gather, whether the library packs it)"""
    lib = ctypes.CDLL(os.path.join(PKG, "liblulesh_host.so"))
    lib.lulesh_host_lmesh_sectors.restype = ctypes.c_double
    lib.lulesh_host_lmesh_sectors.argtypes = [ctypes.c_char_p, ctypes.POINTER(ctypes.c_int)]
    path, packed = str(tmp_path / "rule.lmesh"), ctypes.c_int(-1)
    lmesh.write(path, mesh)
    sectors = lib.lulesh_host_lmesh_sectors(path.encode(), ctypes.byref(packed))
    assert sectors > 0.0
    return sectors, packed.value == 1


def count(mesh):
    n = [len(set(mesh.nodelist[e:e + 32, k] // 4)) for k in range(8)
         for e in range(0, mesh.num_elem, 32)]
    return sum(n) / len(n)


@pytest.mark.parametrize("mesh", [lmesh.box(1), lmesh.box(9), shuffled(2), shuffled(5), shuffled(9),
                                  islands(3), islands(33)])
def test_sectors(tmp_path, mesh):
    sectors, packed = rule(tmp_path, mesh)
    assert sectors == count(mesh)
    assert packed == (sectors >= 28.0)


@pytest.mark.parametrize("nx,packed", [(1, False), (2, False), (3, False), (5, False), (6, False),
                                       (7, True), (8, True), (12, True), (13, True), (17, True)])
def test_shuffled_boxes(tmp_path, nx, packed):
    assert rule(tmp_path, shuffled(nx))[1] == packed


@pytest.mark.parametrize("n,packed", [(1, False), (27, False), (28, True), (31, True), (32, True),
                                      (33, False), (60, True), (127, True), (128, True),
                                      (156, True), (256, True)])
def test_islands(tmp_path, n, packed):
    assert rule(tmp_path, islands(n))[1] == packed
