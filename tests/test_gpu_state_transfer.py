"""State transfers: small states in pinned host memory are read and written by the kernels themselves,
others go through the copy engines.  Both give the same arrays and the same run, whatever the memory is
and wherever the arrays lie in it."""
import numpy as np
import pytest
import torch

from cases import CASES, STATE_KEYS, perturbed_state, prepared
from euler3d_b200 import _lib, meshgen as mg
from euler3d_b200.solver import EulerSolver, FlowConfig, Mesh

pytestmark = pytest.mark.gpu


def buffers(kind, size):
    """Eight arrays of `size` doubles: pageable; pinned one by one; views of one pinned block at odd
    offsets; a pinned block with one pageable array among them; views of a pinned block that overlap the
    block's end by nothing."""
    if kind == "pageable":
        return [np.empty(size) for _ in range(8)], None
    if kind == "pinned":
        t = [torch.empty(size, dtype=torch.float64).pin_memory() for _ in range(8)]
        return [x.numpy() for x in t], t
    t = torch.empty(8 * (size + 3) + 1, dtype=torch.float64).pin_memory()
    flat = t.numpy()
    views = [flat[1 + k * (size + 3):1 + k * (size + 3) + size] for k in range(8)]
    if kind == "mixed":
        views[3] = np.empty(size)
    if kind == "end":
        views[7] = flat[flat.size - size:]
    return views, t


@pytest.mark.parametrize("kind", ["pageable", "pinned", "views", "mixed", "end"])
@pytest.mark.parametrize("precision", [_lib.PREC_FP64_EXACT, _lib.PREC_FP64, _lib.PREC_FP32_FLUX])
@pytest.mark.parametrize("name", ["ogrid", "tets", "large"])
def test_same_state_from_any_memory(name, precision, kind):
    if name == "large":  # above the size that goes directly
        arrays, flow = Mesh.from_raw(mg.bump_box_tets(26)).arrays(), FlowConfig(mach=0.5, precision=precision,
                                                                               ordering=_lib.ORDER_SPATIAL)
    else:
        arrays, flow = prepared(name), CASES[name].flow(precision=precision, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 3, amp=0.02)
    ref = EulerSolver(arrays, flow, autotune=False)
    ref.set_state({k: v.copy() for k, v in state.items()})
    before = ref.get_state()
    ref.run(2)
    after = ref.get_state()
    ref.close()

    s = EulerSolver(arrays, flow, autotune=False)
    inp, keep = buffers(kind, s.state_size)
    out, keep2 = buffers(kind, s.state_size)
    for v, k in zip(inp, STATE_KEYS):
        v[:] = state[k]
    s.set_state(dict(zip(STATE_KEYS, inp)))
    got = s.get_state(dict(zip(STATE_KEYS, out)))
    for k in STATE_KEYS:
        assert np.array_equal(got[k], before[k]), k
    if precision != _lib.PREC_FP32_FLUX:  # its state is the conservative one
        for k in STATE_KEYS:
            assert np.array_equal(got[k], state[k]), k
    s.run(2)
    got = s.get_state(dict(zip(STATE_KEYS, out)))
    for k in STATE_KEYS:
        assert np.array_equal(got[k], after[k]), k
    s.close()


def test_freestream_and_overlapping_outputs():
    """set_freestream is the state a new solver starts from; outputs that share memory are written in
    order (the last array's values stay)."""
    arrays, flow = prepared("channel"), CASES["channel"].flow(precision=_lib.PREC_FP64)
    s = EulerSolver(arrays, flow, autotune=False)
    first = s.get_state()
    n = int(arrays["n_cells"])
    g, u = 1.4, 0.5 * np.sqrt(1.4)
    want = {"rho": 1.0, "u": u, "v": 0.0, "w": 0.0, "p": 1.0, "E": 1 / (g - 1) + u * u / 2}
    for k, v in want.items():
        assert np.allclose(first[k], v, rtol=1e-15, atol=0), k
    s.run(3)
    s.set_freestream()
    again = s.get_state()
    for k in STATE_KEYS:
        assert np.array_equal(first[k], again[k]), k
    t = torch.empty(s.state_size, dtype=torch.float64).pin_memory().numpy()
    s.get_state({k: t for k in STATE_KEYS})
    assert np.array_equal(t[:n], first["M"][:n])
    s.close()


def test_add_and_remove_without_a_step():
    """A solver taken out of a batch before its first step runs on as if it had not been in it."""
    from euler3d_b200.batch import Batch

    arrays, flow = prepared("tets"), CASES["tets"].flow(precision=_lib.PREC_FP64)
    state = perturbed_state(arrays, flow, 5, amp=0.02)
    a, b = (EulerSolver(arrays, flow, autotune=False) for _ in range(2))
    batch = Batch()
    a.set_state(state)
    b.set_state(state)
    batch.add(a, 10)
    batch.remove(a)
    a.run(4)
    b.run(4)
    ga, gb = a.get_state(), b.get_state()
    for k in STATE_KEYS:
        assert np.array_equal(ga[k], gb[k]), k
    batch.close()
