"""FP64 mode's restructured fluxes against the oracle's residual on states that reach their branches.

The Roe flux takes its weights from one root and applies Harten's fix only where a comparison without
a root says so; a symmetry face's flux is the normal force its mirror symmetry leaves.  The states
below put the normal velocity on either side of the sound speed at interior and symmetry faces, and
near it, so that every branch is taken.

Tolerance: a flux component is a sum of about 20 products of roots, reciprocals (each within 2 units
in the last place) and states, so each term carries at most about 50 roundings of 1.1e-16; forming
c~^2 = (gamma - 1)(H - q^2 / 2) loses a factor of H / c^2 < 10 on these states.  That is 6e-14 of the
sum of the terms' sizes, which rho (|u| + c) (1, |u| + c, H) S per face bounds from above to within a
factor of about three: 2e-13.
"""
import numpy as np
import pytest

import pyoracle as po
from cases import CASES, perturbed_state, prepared
from euler3d_b200 import _lib
from euler3d_b200.solver import EulerSolver

pytestmark = pytest.mark.gpu


def shaken(arrays, flow, seed, amp):
    s = perturbed_state(arrays, flow, seed)
    rng = np.random.default_rng(seed + 1)
    c = np.sqrt(flow.gamma * s["p"] / s["rho"])
    for k in "uvw":
        s[k] = amp * c * rng.uniform(-1.0, 1.0, c.size)
    q2 = s["u"] ** 2 + s["v"] ** 2 + s["w"] ** 2
    s["E"] = s["p"] / ((flow.gamma - 1) * s["rho"]) + q2 / 2.0
    s["H"] = s["E"] + s["p"] / s["rho"]
    n = int(arrays["n_cells"])
    s["M"][:n] = c[:n] / np.sqrt(q2[:n])
    return s


@pytest.mark.parametrize("kernel", [1, 5])
@pytest.mark.parametrize("scheme", [_lib.SCHEME_ROE, _lib.SCHEME_AUSM])
@pytest.mark.parametrize("amp", [0.02, 1.1, 2.0])
@pytest.mark.parametrize("name", ["channel", "ogrid", "tets", "pyramids"])
def test_residual_in_every_branch(name, amp, scheme, kernel):
    arrays = prepared(name)
    flow = CASES[name].flow(scheme=scheme, precision=_lib.PREC_FP64, ordering=_lib.ORDER_SPATIAL)
    state = shaken(arrays, flow, 7, amp)
    solver = EulerSolver(arrays, flow, autotune=False)
    solver.run(0, stage_kernel=kernel)  # the kernel that the residual call then uses
    solver.set_state(state)
    got, dt = solver.residual()
    solver.close()

    mesh = po.Mesh(arrays)
    fl = po.flow(flow.mach, flow.aoa, flow.gamma, flow.cfl, scheme=scheme)
    st = po.State(mesh, state)
    po.update_bc(mesh, fl, st)
    want, want_dt = po.compute_residual(mesh, fl, st), po.time_step(mesh, fl, st)

    f2c, area = arrays["face2cell"].reshape(-1, 2), arrays["face_area"]
    a = st.a
    # sizes only: the boundary conditions leave some ghosts of these states with a negative pressure
    speed = np.sqrt(a["u"] ** 2 + a["v"] ** 2 + a["w"] ** 2) + np.sqrt(np.abs(flow.gamma * a["p"] / a["rho"]))
    size = np.abs(np.stack([a["rho"] * speed, *(3 * [a["rho"] * speed ** 2]), a["rho"] * speed * a["H"]], 1))
    per_face = np.maximum(size[f2c[:, 0]], size[f2c[:, 1]]) * area[:, None]
    n, fi = int(arrays["n_cells"]), int(arrays["n_faces_int"])
    scale = np.zeros((n, 5))
    np.add.at(scale, f2c[:, 0], per_face)
    np.add.at(scale, f2c[:fi, 1], per_face[:fi])
    assert np.max(np.abs(got - want) / scale) < 2e-13
    assert np.max(np.abs(dt - want_dt) / want_dt) < 1e-14
