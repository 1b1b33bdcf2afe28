"""Cells of more faces than the element types have (six), which a mesh descriptor may hold: cells of a
prepared mesh merged in pairs.

In the double modes every kernel sums a cell's faces in the same order, so states and RMS are compared
bit for bit with the per-cell gather kernel, and FP64_EXACT with the oracle.  FP32_FLUX has face-tile
kernels only: its residual is compared with the oracle's within the bound of test_gpu_fast_flux.py taken
from double to single rounding, 2e-13 x 2^29 = 1.1e-4 of the sizes of a cell's face terms; a face that is
left out is of the order of one of them.
"""
import numpy as np
import pytest

import pyoracle as po
from cases import CASES, STATE_KEYS, perturbed_state, prepared
from euler3d_b200 import _lib
from euler3d_b200.batch import Batch
from euler3d_b200.solver import EulerSolver

pytestmark = pytest.mark.gpu


def merged(a, seed, pairs):
    """The mesh with `pairs` random pairs of neighbouring cells joined, in the reference's numbering."""
    n, fi, f = int(a["n_cells"]), int(a["n_faces_int"]), int(a["n_faces"])
    f2c = a["face2cell"].reshape(-1, 2)
    group = np.arange(n)
    free = np.ones(n, bool)
    for k in np.random.default_rng(seed).permutation(fi):
        l, r = f2c[k]
        if pairs and free[l] and free[r]:
            group[max(l, r)] = min(l, r)
            free[[l, r]] = False
            pairs -= 1
    kept = group == np.arange(n)
    new = (np.cumsum(kept) - 1)[group]
    cells = int(kept.sum())
    face = np.ones(f, bool)
    face[:fi] = new[f2c[:fi, 0]] != new[f2c[:fi, 1]]
    face_id = np.cumsum(face) - 1
    fi_new = int(face[:fi].sum())
    out = {"n_cells": cells, "n_faces": int(face.sum()), "n_faces_int": fi_new}
    g = np.empty_like(f2c)
    g[:, 0] = new[f2c[:, 0]]
    g[:fi, 1] = new[f2c[:fi, 1]]
    g[fi:, 1] = cells + face_id[fi:] - fi_new
    out["face2cell"] = np.ascontiguousarray(g[face], np.int32).ravel()
    for k, w in (("face_unit_normal", 3), ("face_normal", 3), ("face_center", 3), ("face_area", 1)):
        out[k] = np.ascontiguousarray(np.asarray(a[k]).reshape(-1, w)[face]).ravel()
    out["cell_volume"] = np.zeros(cells)
    np.add.at(out["cell_volume"], new, a["cell_volume"])
    lists = [[] for _ in range(cells)]
    for c in range(n):
        for k in a["cell2face"][a["cell2face_ptr"][c]:a["cell2face_ptr"][c + 1]]:
            if face[k]:
                lists[new[c]].append(face_id[k])
    out["cell2face_ptr"] = np.concatenate([[0], np.cumsum([len(x) for x in lists])]).astype(np.int32)
    out["cell2face"] = np.concatenate(lists).astype(np.int32)
    for tag in ("wall", "farfield", "sym"):
        faces = face_id[a[f"{tag}_face"]].astype(np.int32)
        out[f"{tag}_face"] = faces
        out[f"{tag}_interior"] = new[a[f"{tag}_interior"]].astype(np.int32)
        out[f"{tag}_ghost"] = (cells + faces - fi_new).astype(np.int32)
    return out


def case(name):
    arrays = merged(prepared(name), 3, 20)
    most = int(np.diff(arrays["cell2face_ptr"]).max())
    assert most >= 7
    return arrays


def run(arrays, flow, state, kernel):
    s = EulerSolver(arrays, flow, autotune=False)
    s.set_state(state)
    s.run(5, stage_kernel=kernel)
    out = s.get_state(), s.rms_history()
    s.close()
    return out


@pytest.mark.parametrize("precision", [_lib.PREC_FP64_EXACT, _lib.PREC_FP64])
@pytest.mark.parametrize("name", ["channel", "ogrid", "pyramids"])
def test_double_modes(name, precision):
    arrays = case(name)
    flow = CASES[name].flow(precision=precision, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 4)
    want = run(arrays, flow, state, _lib.KERNEL_GATHER)
    kernels = [_lib.KERNEL_AUTO, _lib.KERNEL_TILE, _lib.KERNEL_TILE_PIPE]
    for kernel in kernels + ([_lib.KERNEL_TILE_B3] if precision == _lib.PREC_FP64 else []):
        got = run(arrays, flow, state, kernel)
        assert np.array_equal(got[1], want[1]), kernel
        for k in STATE_KEYS:
            assert np.array_equal(got[0][k], want[0][k]), (kernel, k)
    for kernel in (_lib.BATCH_KERNEL_TILES, _lib.BATCH_KERNEL_WS):
        s, b = EulerSolver(arrays, flow, autotune=False), Batch()
        s.set_state(state)
        b.set_kernel(kernel)
        b.add(s, 5)
        b.run_all()
        got = s.get_state()
        b.close()
        s.close()
        for k in STATE_KEYS:
            assert np.array_equal(got[k], want[0][k]), (kernel, k)
    if precision == _lib.PREC_FP64_EXACT:
        mesh = po.Mesh(arrays)
        o = po.State(mesh, state)
        po.run(mesh, po.flow(flow.mach, flow.aoa, flow.gamma, flow.cfl), o, 5)
        for k in ("rho", "u", "v", "w", "p"):
            assert np.array_equal(want[0][k], o.a[k]), k


@pytest.mark.parametrize("kernel", [_lib.KERNEL_TILE, _lib.KERNEL_TILE_PIPE, _lib.KERNEL_TILE_B3])
@pytest.mark.parametrize("name", ["channel", "ogrid", "pyramids"])
def test_single_precision_fluxes(name, kernel):
    arrays = case(name)
    flow = CASES[name].flow(precision=_lib.PREC_FP32_FLUX, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 4)
    s = EulerSolver(arrays, flow, autotune=False)
    s.run(0, stage_kernel=kernel)
    s.set_state(state)
    got, _ = s.residual()
    s.close()
    mesh = po.Mesh(arrays)
    st = po.State(mesh, state)
    fl = po.flow(flow.mach, flow.aoa, flow.gamma, flow.cfl)
    po.update_bc(mesh, fl, st)
    want, a = po.compute_residual(mesh, fl, st), st.a
    speed = np.sqrt(a["u"] ** 2 + a["v"] ** 2 + a["w"] ** 2) + np.sqrt(np.abs(flow.gamma * a["p"] / a["rho"]))
    size = np.abs(np.stack([a["rho"] * speed, *(3 * [a["rho"] * speed ** 2]), a["rho"] * speed * a["H"]], 1))
    f2c, fi = arrays["face2cell"].reshape(-1, 2), arrays["n_faces_int"]
    per_face = np.maximum(size[f2c[:, 0]], size[f2c[:, 1]]) * arrays["face_area"][:, None]
    scale = np.zeros((arrays["n_cells"], 5))
    np.add.at(scale, f2c[:, 0], per_face)
    np.add.at(scale, f2c[:fi, 1], per_face[:fi])
    assert np.max(np.abs(got - want) / scale) < 1.1e-4


@pytest.mark.parametrize("precision", [_lib.PREC_FP64_EXACT, _lib.PREC_FP64, _lib.PREC_FP32_FLUX])
def test_joining_and_leaving_a_batch(precision):
    """A member with such cells joins a running batch of ordinary ones and leaves it: every member computes
    what it computes alone."""
    def solver(arrays, name):
        flow = CASES[name].flow(precision=precision, ordering=_lib.ORDER_SPATIAL)
        s = EulerSolver(arrays, flow, autotune=False)
        s.set_state(perturbed_state(arrays, flow, 4))
        return s

    meshes = [(prepared("tets"), "tets", 24), (case("channel"), "channel", 6), (prepared("ogrid"), "ogrid", 12)]
    want = []
    for arrays, name, n in meshes:
        s = solver(arrays, name)
        s.run(n, stage_kernel=_lib.KERNEL_TILE)
        want.append((s.get_state(), s.rms_history()))
        s.close()
    b = Batch()
    members = [solver(arrays, name) for arrays, name, _ in meshes]
    b.add(members[0], 24)
    b.step(4)
    b.add(members[1], 6)
    b.step(4)
    b.add(members[2], 12)
    b.run_all(4)
    for s, (state, history) in zip(members, want):
        assert np.array_equal(s.rms_history(), history)
        got = s.get_state()
        for k in STATE_KEYS:
            assert np.array_equal(got[k], state[k]), k
    b.close()
