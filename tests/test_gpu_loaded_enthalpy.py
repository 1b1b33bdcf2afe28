"""States whose total enthalpy and energy do not follow from density, pressure and velocity: set_state takes
all eight arrays, and the reference computes with them as they are until its first update.  The ghosts'
enthalpies do follow, so a symmetry face has two different ones on its sides.

The FP64 mode's residual against the oracle's, within the bound of test_gpu_fast_flux.py (2e-13 of the
sizes of a cell's face terms, which the enthalpy enters), and the run that follows against FP64_EXACT
within 1e-10."""
import numpy as np
import pytest

import pyoracle as po
from cases import CASES, perturbed_state, prepared
from euler3d_b200 import _lib
from euler3d_b200.solver import EulerSolver

pytestmark = pytest.mark.gpu


def loaded(arrays, flow, off):
    s = perturbed_state(arrays, flow, 5)
    rng = np.random.default_rng(6)
    f = 1.0 + off * rng.uniform(-1.0, 1.0, s["H"].size)
    s["H"] *= f
    s["E"] *= f
    return s


@pytest.mark.parametrize("kernel", [_lib.KERNEL_GATHER, _lib.KERNEL_TILE, _lib.KERNEL_TILE_PIPE, _lib.KERNEL_TILE_B3,
                                    _lib.KERNEL_COLOUR])
@pytest.mark.parametrize("scheme", [_lib.SCHEME_ROE, _lib.SCHEME_AUSM])
@pytest.mark.parametrize("off", [1e-6, 0.1])
@pytest.mark.parametrize("name", ["channel", "ogrid", "tets"])
def test_residual(name, off, scheme, kernel):
    arrays = prepared(name)
    flow = CASES[name].flow(scheme=scheme, precision=_lib.PREC_FP64, ordering=_lib.ORDER_SPATIAL)
    state = loaded(arrays, flow, off)
    s = EulerSolver(arrays, flow, autotune=False)
    s.run(0, stage_kernel=kernel)
    s.set_state(state)
    got, _ = s.residual()
    s.close()
    mesh = po.Mesh(arrays)
    fl = po.flow(flow.mach, flow.aoa, flow.gamma, flow.cfl, scheme=scheme)
    st = po.State(mesh, state)
    po.update_bc(mesh, fl, st)
    want, a = po.compute_residual(mesh, fl, st), st.a
    speed = np.sqrt(a["u"] ** 2 + a["v"] ** 2 + a["w"] ** 2) + np.sqrt(np.abs(flow.gamma * a["p"] / a["rho"]))
    size = np.abs(np.stack([a["rho"] * speed, *(3 * [a["rho"] * speed ** 2]), a["rho"] * speed * a["H"]], 1))
    f2c, fi = arrays["face2cell"].reshape(-1, 2), int(arrays["n_faces_int"])
    per_face = np.maximum(size[f2c[:, 0]], size[f2c[:, 1]]) * arrays["face_area"][:, None]
    scale = np.zeros((int(arrays["n_cells"]), 5))
    np.add.at(scale, f2c[:, 0], per_face)
    np.add.at(scale, f2c[:fi, 1], per_face[:fi])
    assert np.max(np.abs(got - want) / scale) < 2e-13


@pytest.mark.parametrize("kernel", [_lib.KERNEL_AUTO, _lib.KERNEL_TILE_B3])
@pytest.mark.parametrize("integrator", [_lib.INTEGRATOR_RK5, _lib.INTEGRATOR_EULER])
def test_run(integrator, kernel):
    arrays = prepared("channel")
    out = []
    for precision in (_lib.PREC_FP64_EXACT, _lib.PREC_FP64):
        flow = CASES["channel"].flow(precision=precision, integrator=integrator, ordering=_lib.ORDER_SPATIAL)
        s = EulerSolver(arrays, flow, autotune=False)
        s.set_state(loaded(arrays, flow, 0.05))
        s.run(3, stage_kernel=kernel if precision == _lib.PREC_FP64 else _lib.KERNEL_AUTO)
        out.append(s.get_state())
        s.close()
    for k in ("rho", "u", "v", "w", "p"):
        assert np.max(np.abs(out[0][k] - out[1][k])) < 1e-10 * np.max(np.abs(out[0][k])), k
