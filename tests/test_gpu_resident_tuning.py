"""Where more than three tiles share an SM, creating a tuned solver times the resident kernel against the
stage kernels: the solver it leaves is a new one (freestream, no history, no coefficients), whichever way
its runs take, and they give the bits of an untuned solver's."""
import numpy as np
import pytest

from cases import STATE_KEYS, perturbed_state
from euler3d_b200 import _lib, meshgen as mg
from euler3d_b200.solver import EulerSolver, FlowConfig, Mesh

pytestmark = pytest.mark.gpu
_meshes = {}


@pytest.mark.parametrize("integrator", [_lib.INTEGRATOR_RK5, _lib.INTEGRATOR_EULER])
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_FP32_FLUX])
@pytest.mark.parametrize("cells", [23, 25])  # four tiles per SM, five
def test_tuned_solver_is_new(cells, precision, integrator):
    if precision == _lib.PREC_FP32_FLUX and integrator == _lib.INTEGRATOR_EULER:
        pytest.skip("FP32_FLUX runs RK5 only")
    if cells not in _meshes:
        _meshes[cells] = Mesh.from_raw(mg.bump_box_tets(cells)).arrays()
    arrays = _meshes[cells]
    flow = FlowConfig(mach=0.5, aoa=1.0, cfl=0.6, precision=precision, integrator=integrator,
                      ordering=_lib.ORDER_SPATIAL)
    out = []
    for tuned in (True, False):
        s = EulerSolver(arrays, flow, autotune=tuned)
        new = [s.get_state(), s.rms_history(), s.coefficient_history(), s.wall_cp(), np.concatenate(s.coefficients())]
        first = s.run(3)
        states = [s.get_state()]
        s.set_state(perturbed_state(arrays, flow, 3))
        last = s.run(5)
        states.append(s.get_state())
        out.append((new, first, last, states, s.rms_history()))
        s.close()
    a, b = out
    assert a[0][1].size == a[0][2].size == 0 and not a[0][3].any()
    for k in STATE_KEYS:
        assert np.array_equal(a[0][0][k], b[0][0][k])
        for i in (0, 1):
            assert np.array_equal(a[3][i][k], b[3][i][k]), (i, k)
    assert np.array_equal(a[0][4], b[0][4]) and np.array_equal(a[4], b[4])
    for i in (1, 2):
        for k in ("iterations", "n_rms", "last_rms", "force", "moment"):
            assert a[i][k] == b[i][k], k
    assert b[1]["kernel_launches"] == 1  # untuned: the resident kernel


def test_exact_mode():
    """Its control block sums sequentially: with four tiles per SM a resident iteration takes nearly twice
    as long as one of stage kernels, and the tuned solver runs those."""
    got = []
    for cells in (18, 22):  # 274 and 500 tiles
        arrays = Mesh.from_raw(mg.bump_box_tets(cells)).arrays()
        flow = FlowConfig(mach=0.5, cfl=0.6, precision=_lib.PREC_FP64_EXACT, ordering=_lib.ORDER_SPATIAL)
        s = EulerSolver(arrays, flow)
        got.append(s.run(2)["kernel_launches"] == 1)
        s.close()
    assert got == [True, False]
