"""The resident kernel's waits between its blocks, made to run out by a small poll limit
(``e3d_solver_set_wait_limit``): a tile's wait for its neighbours' cells, for the iteration's decision,
and the control block's for the tiles.  Nothing hangs or faults: every wait has the limit, and a block
whose wait runs out raises the run's fault word and returns.

A run under a limit either reports the timeout or, where no wait was long enough, is the run without the
limit; at one or two polls (about 0.5 us each) the control block's first wait, which lasts a whole
iteration, always runs out.  The solver then goes on as if nothing had happened."""
import numpy as np
import pytest

from cases import STATE_KEYS, perturbed_state
from euler3d_b200 import _lib, meshgen as mg
from euler3d_b200.solver import EulerSolver, FlowConfig, Mesh

pytestmark = pytest.mark.gpu

SIZES = {"two_tiles": lambda: mg.bump_channel(13, 11, 2), "many": lambda: mg.biconvex_ogrid(60, 40, 4, span=0.4),
         "several_per_sm": lambda: mg.bump_box_tets(16)}
_meshes = {}


@pytest.mark.parametrize("precision", [_lib.PREC_FP64_EXACT, _lib.PREC_FP64, _lib.PREC_FP32_FLUX])
@pytest.mark.parametrize("name", list(SIZES))
def test_waits_run_out(name, precision):
    if name not in _meshes:
        _meshes[name] = Mesh.from_raw(SIZES[name]()).arrays()
    arrays = _meshes[name]
    flow = FlowConfig(mach=0.5, cfl=1.0, precision=precision, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 9, amp=0.02)
    s = EulerSolver(arrays, flow, autotune=False)
    s.set_state(state)
    stats = s.run(12, sampling=3)
    assert stats["kernel_launches"] == 1
    want, history = s.get_state(), s.rms_history()

    def is_that_run():
        assert np.array_equal(s.rms_history(), history)
        got = s.get_state()
        for k in STATE_KEYS:
            assert np.array_equal(got[k], want[k]), k

    for polls in (0, 1, 2, 4, 8, 16, 32, 64, 128, 512):
        s.set_wait_limit(polls)
        s.set_state(state)
        try:
            s.run(12, sampling=3)
        except _lib.E3DError as e:
            assert e.status == _lib.E3D_ERR_TIMEOUT
            assert e.stats["iterations"] < 12
        else:
            assert polls > 2
            is_that_run()
    s.set_wait_limit(-1)
    s.set_state(state)
    s.run(12, sampling=3)
    is_that_run()
    s.close()
