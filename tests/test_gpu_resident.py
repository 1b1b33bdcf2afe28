"""The resident kernel (whole iterations in one launch, one block per face tile) against the stage
kernels, which every other test pins to the oracle.

Both run the same device functions on the same cells in the same order, so states, RMS history,
coefficients, counters and stop reasons are compared bit for bit: meshes of one tile and of several,
with a ragged last tile, with as many tiles as several blocks per SM hold, every precision, scheme and
integrator, every stop test, odd and even iteration counts and several launches per run.
"""
import threading

import numpy as np
import pytest

from cases import CASES, STATE_KEYS, perturbed_state, prepared
from euler3d_b200 import _lib, meshgen as mg
from euler3d_b200.solver import EulerSolver, FlowConfig, Mesh

pytestmark = pytest.mark.gpu

PRECISIONS = [_lib.PREC_FP64_EXACT, _lib.PREC_FP64, _lib.PREC_FP32_FLUX]
SIZES = {  # tiles: 1, 1 (ragged), 3, 32, 148+, about 450, about 740 of tetrahedra
    "one_tile": lambda: mg.bump_channel(8, 8, 2),
    "less_than_a_tile": lambda: mg.bump_channel(5, 5, 2),
    "ragged": lambda: mg.bump_box_tets(4),
    "c1": lambda: mg.bump_channel(),
    "one_per_sm": lambda: mg.bump_channel(99, 97, 2),
    "ogrid_three_per_sm": lambda: mg.biconvex_ogrid(120, 60, 4, span=0.4),
    "tets_five_per_sm": lambda: mg.bump_box_tets(25),
}
_meshes = {}


def mesh(name):
    if name not in _meshes:
        _meshes[name] = Mesh.from_raw(SIZES[name]()).arrays() if name in SIZES else prepared(name)
    return _meshes[name]


def both(arrays, flow, state, **run):
    """The same run with the resident kernel and with the stage kernels in CUDA graphs."""
    out = []
    for kernel in (0, _lib.KERNEL_TILE):
        s = EulerSolver(arrays, flow, autotune=False)
        s.set_state(state)
        stats = s.run(stage_kernel=kernel, **run)
        out.append((stats, s.get_state(), s.rms_history(), s.coefficient_history(), s.wall_cp()))
        s.close()
    return out


def same(a, b):
    for k in ("iterations", "stop_reason", "n_rms", "last_rms", "cl", "cd", "cm", "force", "moment"):
        assert a[0][k] == b[0][k], k
    for k in STATE_KEYS:
        assert np.array_equal(a[1][k], b[1][k]), k
    for i in (2, 3, 4):
        assert np.array_equal(a[i], b[i])


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("name", list(SIZES))
def test_same_bits(name, precision):
    arrays = mesh(name)
    flow = FlowConfig(mach=0.6, aoa=1.0, cfl=0.9, precision=precision, ordering=_lib.ORDER_SPATIAL)
    a, b = both(arrays, flow, perturbed_state(arrays, flow, 3, amp=0.02), max_iter=7)
    same(a, b)
    assert a[0]["iterations"] == 7
    if not (name == "tets_five_per_sm" and precision == _lib.PREC_FP64_EXACT):  # four per SM in that mode
        assert a[0]["kernel_launches"] == 1 < b[0]["kernel_launches"]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("name", ["channel", "channel_supersonic", "ogrid", "tets", "pyramids"])
def test_every_boundary_and_scheme(name, precision):
    arrays = prepared(name)
    for scheme in (_lib.SCHEME_ROE, _lib.SCHEME_AUSM):
        flow = CASES[name].flow(precision=precision, scheme=scheme, ordering=_lib.ORDER_NATIVE)
        state = perturbed_state(arrays, flow, 5)
        same(*both(arrays, flow, state, max_iter=12, sampling=3))


@pytest.mark.parametrize("precision", PRECISIONS[:2])
def test_explicit_euler(precision):
    arrays = prepared("tets")
    flow = FlowConfig(mach=0.6, cfl=0.6, precision=precision, integrator=_lib.INTEGRATOR_EULER,
                      ordering=_lib.ORDER_SPATIAL)
    same(*both(arrays, flow, perturbed_state(arrays, flow, 8), max_iter=9))


@pytest.mark.parametrize("run", [
    dict(max_iter=0), dict(max_iter=1), dict(max_iter=2), dict(max_iter=21, check_every=4),
    dict(max_iter=600, min_residual_drop=1e-2), dict(max_iter=600, min_residual=2e-4),
    dict(max_iter=900, min_aerocoeff_error=2e-4), dict(max_iter=900, min_aerocoeff_error=2e-4, sampling=7),
    dict(max_iter=25, sampling=10), dict(max_iter=900, stall_window=15), dict(max_iter=300, sampling=1000),
], ids=str)
@pytest.mark.parametrize("precision", PRECISIONS)
def test_stop_tests(precision, run):
    arrays = prepared("channel")
    flow = CASES["channel"].flow(precision=precision, ordering=_lib.ORDER_SPATIAL)
    same(*both(arrays, flow, perturbed_state(arrays, flow, 2), **run))


def test_runs_continue_from_either_buffer():
    """Odd runs end in the second state buffer; later runs, residuals and states go on from there."""
    arrays = prepared("ogrid")
    flow = CASES["ogrid"].flow(precision=_lib.PREC_FP64, ordering=_lib.ORDER_SPATIAL)
    out = []
    for kernel in (0, _lib.KERNEL_TILE):
        s = EulerSolver(arrays, flow, autotune=False)
        got = []
        for n in (3, 4, 1, 1, 6):
            s.run(n, stage_kernel=kernel)
            got += [s.residual()[0], s.get_state()["p"], np.concatenate(s.coefficients())]
        out.append(got)
        s.close()
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_nonfinite_stops():
    arrays = prepared("channel")
    flow = FlowConfig(mach=0.5, cfl=60.0, precision=_lib.PREC_FP64, ordering=_lib.ORDER_SPATIAL)
    seen = []
    for kernel in (0, _lib.KERNEL_TILE):
        s = EulerSolver(arrays, flow, autotune=False)
        s.set_state(perturbed_state(arrays, flow, 4))
        with pytest.raises(_lib.E3DError) as e:
            s.run(500, stage_kernel=kernel)
        assert e.value.status == _lib.E3D_ERR_NONFINITE
        seen.append((e.value.stats["iterations"], e.value.stats["n_rms"]))
        s.set_freestream()
        assert s.run(0)["iterations"] == 0
        s.close()
    assert seen[0] == seen[1]


@pytest.mark.parametrize("precision", PRECISIONS)
def test_timeout_stops_and_recovers(precision):
    """Every tile's first wait gives up at once (its copies still land); the run reports the timeout
    and the solver goes on as if nothing had happened."""
    arrays = prepared("ogrid")
    flow = CASES["ogrid"].flow(precision=precision, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 6)
    s = EulerSolver(arrays, flow, autotune=False)
    s.set_state(state)
    s.set_wait_limit(0)
    with pytest.raises(_lib.E3DError) as e:
        s.run(20)
    assert e.value.status == _lib.E3D_ERR_TIMEOUT
    assert e.value.stats["iterations"] == 0 and e.value.stats["n_rms"] == 0
    s.set_wait_limit(-1)
    s.set_state(state)
    s.run(5)
    got = s.get_state()
    s.close()
    want = both(arrays, flow, state, max_iter=5)[1][1]
    for k in STATE_KEYS:
        assert np.array_equal(got[k], want[k]), k


def test_two_threads():
    """Solvers run from several threads at once: one resident run at a time, the others on the stage
    kernels, the same bits."""
    arrays = mesh("one_per_sm")
    flow = FlowConfig(mach=0.5, cfl=1.0, precision=_lib.PREC_FP64, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 9, amp=0.02)
    want = both(arrays, flow, state, max_iter=40)[1]
    got = [None] * 3

    def work(i):
        s = EulerSolver(arrays, flow, autotune=False)
        for _ in range(4):
            s.set_state(state)
            s.run(40)
        got[i] = (s.get_state(), s.rms_history())
        s.close()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for st, hist in got:
        assert np.array_equal(hist, want[2])
        for k in STATE_KEYS:
            assert np.array_equal(st[k], want[1][k]), k


@pytest.mark.parametrize("kind", ["freestream", "one_cell", "random", "wide"])
@pytest.mark.parametrize("name", ["channel", "tets", "one_per_sm", "ogrid_three_per_sm"])
def test_exact_rms_is_the_sequential_sum(name, kind):
    """FP64_EXACT's RMS is the reference's running sum over the cells: rounding-noise residuals with
    many equal values and zeros (freestream), a few large ones among zeros, residuals of one size and
    residuals over many decades, checked against that sum of the residual the solver returns."""
    arrays = mesh(name)
    flow = FlowConfig(mach=0.5, aoa=1.0, cfl=1.0, precision=_lib.PREC_FP64_EXACT, ordering=_lib.ORDER_SPATIAL,
                      integrator=_lib.INTEGRATOR_EULER)
    s = EulerSolver(arrays, flow, autotune=False)
    n = int(arrays["n_cells"])
    state = s.get_state()
    rng = np.random.default_rng(1)
    if kind == "one_cell":
        state["rho"][n // 2] *= 1.01
    elif kind == "random":
        state["rho"][:n] *= 1.0 + 0.01 * rng.uniform(-1, 1, n)
    elif kind == "wide":
        state["rho"][:n] *= 1.0 + 10.0 ** rng.uniform(-15, -2, n)
    s.set_state(state)
    r = s.residual()[0][:, 0]
    for kernel in (0, _lib.KERNEL_TILE):
        s.set_state(state)
        s.run(1, stage_kernel=kernel)  # explicit Euler: the RMS is this residual's
        total = 0.0
        for v in (r * r).tolist():
            total += v
        assert s.rms_history()[0] == np.sqrt(total / n)
    s.close()


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("run", [
    dict(max_iter=1), dict(max_iter=2), dict(max_iter=7, check_every=4), dict(max_iter=8, check_every=4),
    dict(max_iter=40, sampling=3), dict(max_iter=33, sampling=11), dict(max_iter=64), dict(max_iter=21, sampling=22),
    dict(max_iter=400, min_residual_drop=3e-2), dict(max_iter=900, min_aerocoeff_error=2e-4),
], ids=str)
@pytest.mark.parametrize("name", ["ogrid", "c1"])
def test_forces_in_the_first_stage(name, run, precision):
    """Force coefficients that cannot stop the run are integrated beside the next iteration's first
    stage (or after the last one): the same samples, wall Cp and stop as with a kernel of their own
    after every iteration, which the timed runs keep."""
    arrays = mesh(name)
    flow = FlowConfig(mach=0.5, aoa=1.0, cfl=1.0, precision=precision, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 12, amp=0.02)
    out = []
    for profile in (0, 1):
        s = EulerSolver(arrays, flow, autotune=False)
        s.set_state(state)
        stats = s.run(stage_kernel=_lib.KERNEL_TILE, profile_stages=profile, **run)
        out.append((stats, s.get_state(), s.rms_history(), s.coefficient_history(), s.wall_cp()))
        s.close()
    same(*out)
