"""The cell order behind E3D_ORDER_SPATIAL (euler3d_b200/csrc/tile_order.hpp), compiled for the CPU."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from cases import prepared
from euler3d_b200 import meshgen as mg
from euler3d_b200.solver import Mesh

HERE = os.path.dirname(os.path.abspath(__file__))
SOURCE = """
#include "tile_order.hpp"
extern "C" void order_cells(int n, int n_int, const int *f2c, const double *normal, const double *centre, int tile, int *out) {
    std::vector<double> x(centre, centre + 3 * (size_t)n);
    auto o = e3d::compact_tile_order(n, n_int, f2c, normal, x, tile);
    std::copy(o.begin(), o.end(), out);
}
"""


@pytest.fixture(scope="module")
def order_cells(tmp_path_factory):
    d = tmp_path_factory.mktemp("order")
    (d / "order.cpp").write_text(SOURCE)
    inc = os.path.join(os.path.dirname(HERE), "euler3d_b200", "csrc")
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-shared", "-fPIC", f"-I{inc}", "-o", str(d / "order.so"),
                    str(d / "order.cpp")], check=True)
    fn = C.CDLL(str(d / "order.so")).order_cells

    def call(a, centre, tile):
        p = lambda v, t: np.ascontiguousarray(v, t).ctypes.data_as(C.c_void_p)  # noqa: E731
        out = np.empty(int(a["n_cells"]), np.int32)
        keep = [np.ascontiguousarray(v, t) for v, t in ((a["face2cell"], np.int32), (a["face_unit_normal"], np.float64),
                                                        (centre, np.float64))]
        fn(out.size, int(a["n_faces_int"]), p(keep[0], np.int32), p(keep[1], np.float64), p(keep[2], np.float64), tile,
           out.ctypes.data_as(C.c_void_p))
        return out

    return call


def cut_faces(a, order, tile):
    where = np.empty(order.size, np.int64)
    where[order] = np.arange(order.size) // tile
    f = a["face2cell"].reshape(-1, 2)[: int(a["n_faces_int"])]
    return int((where[f[:, 0]] != where[f[:, 1]]).sum())


@pytest.mark.parametrize("name", ["channel", "ogrid", "tets", "pyramids"])
@pytest.mark.parametrize("tile", [1, 7, 64, 128, 100000])
def test_is_a_permutation_and_repeatable(order_cells, name, tile):
    a = prepared(name)
    first, again = (order_cells(a, a["cell_centroid"], tile) for _ in range(2))
    assert np.array_equal(np.sort(first), np.arange(first.size)) and np.array_equal(first, again)


def test_degenerate_geometry(order_cells):
    """Coincident centres and faces without a normal still give an order."""
    a = dict(prepared("tets"))
    a["face_unit_normal"] = np.full_like(a["face_unit_normal"], np.nan)
    o = order_cells(a, np.zeros_like(a["cell_centroid"]), 16)
    assert np.array_equal(np.sort(o), np.arange(o.size))


def test_threads_and_compactness(order_cells):
    """A mesh large enough for the threads: repeatable, and far fewer cut faces than the mesh's own order."""
    a = Mesh.from_raw(mg.biconvex_ogrid(96, 64, 4, span=0.4)).arrays()
    first, again = (order_cells(a, a["cell_centroid"], 128) for _ in range(2))
    assert np.array_equal(first, again) and np.array_equal(np.sort(first), np.arange(first.size))
    assert cut_faces(a, first, 128) < 0.5 * cut_faces(a, np.arange(first.size), 128)


@pytest.mark.parametrize("offset", [0.0, 1e3])
@pytest.mark.parametrize("nx,ny", [(100, 100), (700, 600)])
def test_one_layer(order_cells, nx, ny, offset):
    """A grid one cell thick, numbered at random, flat but for rounding in a direction that is no
    coordinate axis's alone.  Square tiles of 128 cells cut 4 sqrt(128) / 2 of their 256 faces, 8.8 %;
    half as much again is allowed."""
    n = nx * ny
    cell = np.random.default_rng(1).permutation(n)
    idx = cell.reshape(ny, nx)
    faces = np.concatenate([np.stack([idx[:, :-1].ravel(), idx[:, 1:].ravel()], 1),
                            np.stack([idx[:-1].ravel(), idx[1:].ravel()], 1)])
    r = np.array([[1.0, 0.0, 0.0], [0.0, 0.6, 0.8], [0.0, -0.8, 0.6]])
    normal = np.concatenate([np.tile(r[0], (ny * (nx - 1), 1)), np.tile(r[1], ((ny - 1) * nx, 1))])
    for axes in (np.eye(3), r):
        x = np.empty((n, 3))
        x[cell] = np.stack([np.tile(np.arange(nx), ny), np.repeat(np.arange(ny), nx), np.zeros(n)], 1) @ axes + offset
        a = {"n_cells": n, "n_faces_int": len(faces), "face2cell": faces.ravel(),
             "face_unit_normal": normal if axes is r else np.tile([1.0, 0.0, 0.0], (len(faces), 1))}
        o = order_cells(a, x, 128)
        assert np.array_equal(np.sort(o), np.arange(n))
        assert cut_faces(a, o, 128) < 1.5 * 0.088 * len(faces)
