"""States with negative densities and pressures, which a run that is about to fail passes through: the
FP64 and FP32_FLUX modes' restructured operations end in a NaN where the reference's do."""
import numpy as np
import pytest

from cases import CASES, perturbed_state, prepared
from euler3d_b200 import _lib
from euler3d_b200.solver import EulerSolver, FlowConfig

pytestmark = pytest.mark.gpu

DOUBLE_KERNELS = [_lib.KERNEL_GATHER, _lib.KERNEL_TILE, _lib.KERNEL_TILE_PIPE, _lib.KERNEL_TILE_B3, _lib.KERNEL_COLOUR]


def negated(state, cells):
    """Density and pressure of `cells` with the other sign, E and H as they were (p / rho is)."""
    out = {k: v.copy() for k, v in state.items()}
    for k in ("rho", "p"):
        out[k][cells] *= -1.0
    return out


def residual(arrays, flow, state, kernel):
    s = EulerSolver(arrays, flow, autotune=False)
    s.run(0, stage_kernel=kernel)
    s.set_state(state)
    r, _ = s.residual()
    s.close()
    return r


@pytest.mark.parametrize("kernel", DOUBLE_KERNELS)
@pytest.mark.parametrize("name", ["channel", "ogrid", "tets"])
def test_negative_everywhere(name, kernel):
    arrays = prepared(name)
    flow = dict(mach=0.5, cfl=1.0, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, FlowConfig(**flow), 3)
    state = negated(state, slice(0, int(arrays["n_cells"])))
    assert np.isnan(residual(arrays, FlowConfig(precision=_lib.PREC_FP64_EXACT, **flow), state, _lib.KERNEL_TILE)).all()
    assert np.isnan(residual(arrays, FlowConfig(precision=_lib.PREC_FP64, **flow), state, kernel)).all()


def cube():
    """One unit cube, every face a symmetry face."""
    unit = np.array([[-1, 0, 0], [1, 0, 0], [0, -1, 0], [0, 1, 0], [0, 0, -1], [0, 0, 1]], float)
    f = np.arange(6, dtype=np.int32)
    return {"n_cells": 1, "n_faces": 6, "n_faces_int": 0, "face2cell": np.stack([0 * f, 1 + f], 1).ravel(),
            "face_unit_normal": unit.ravel(), "face_normal": unit.ravel(), "face_area": np.ones(6),
            "face_center": (0.5 + 0.5 * unit).ravel(), "cell_volume": np.ones(1),
            "cell2face_ptr": np.array([0, 6], np.int32), "cell2face": f,
            "sym_face": f, "sym_interior": 0 * f, "sym_ghost": 1 + f}


@pytest.mark.parametrize("kernel", DOUBLE_KERNELS)
@pytest.mark.parametrize("sign", [1, -1])
def test_symmetry_faces_alone(sign, kernel):
    arrays = cube()
    flow = dict(mach=0.5, cfl=1.0)
    state = perturbed_state(arrays, FlowConfig(**flow), 3)
    state = negated(state, slice(0, 1)) if sign < 0 else state
    exact = residual(arrays, FlowConfig(precision=_lib.PREC_FP64_EXACT, **flow), state, _lib.KERNEL_TILE)
    fast = residual(arrays, FlowConfig(precision=_lib.PREC_FP64, **flow), state, kernel)
    assert np.isnan(exact[0, 1:4]).all() == np.isnan(fast[0, 1:4]).all() == (sign < 0)


@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_FP32_FLUX])
@pytest.mark.parametrize("name", ["channel", "ogrid", "tets"])
def test_ghosts_of_negative_cells(name, precision):
    """Ghost records of cells whose density and pressure are both negative (the reference's sound speed
    is a number there), of every boundary kind: the exact mode's, within 30 roundings that the mixed
    signs magnify up to 30 times (2^-53, or 2^-24 of FP32_FLUX's cell states)."""
    arrays = prepared(name)
    n = int(arrays["n_cells"])
    base = perturbed_state(arrays, FlowConfig(mach=0.5), 3)
    cells = np.flatnonzero(np.random.default_rng(5).uniform(size=n) < 0.5)
    got = []
    for prec in (_lib.PREC_FP64_EXACT, precision):
        flow = FlowConfig(mach=0.5, cfl=1.0, precision=prec, ordering=_lib.ORDER_SPATIAL)
        s = EulerSolver(arrays, flow, autotune=False)
        s.set_state(negated(base, cells))
        s.residual()
        got.append(s.get_state())
        s.close()
    tol = 900 * (2.0 ** -53 if precision == _lib.PREC_FP64 else 2.0 ** -24)
    for k in ("rho", "u", "v", "w", "p", "E", "H", "M"):
        want, have = got[0][k][n:], got[1][k][n:]
        assert np.max(np.abs(have - want)) <= tol * np.max(np.abs(want)), k


@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_FP32_FLUX])
def test_ghost_mach_of_a_fluid_at_rest(precision):
    """No velocity and a negative pressure: the ghost's Mach number is 0 / NaN."""
    arrays = cube()
    state = perturbed_state(arrays, FlowConfig(mach=0.5), 3)
    for k in "uvw":
        state[k][:] = 0.0
    state["p"][0] = -1.0
    for prec in (_lib.PREC_FP64_EXACT, precision):
        s = EulerSolver(arrays, FlowConfig(mach=0.5, precision=prec), autotune=False)
        s.set_state(state)
        s.residual()
        assert np.isnan(s.get_state()["M"][1:]).all()
        s.close()


@pytest.mark.parametrize("kernel", DOUBLE_KERNELS)
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("key", ["u", "v", "w", "H"])
def test_ausm_symmetry_faces_pass_on_nan(key, value, kernel):
    """A velocity or an enthalpy that is no finite number: the symmetry faces of its cell, whose splits
    cancel, still end in NaN where the reference's products do (0 x NaN, 0 x inf)."""
    arrays = cube()
    out = []
    for prec, k in ((_lib.PREC_FP64_EXACT, _lib.KERNEL_TILE), (_lib.PREC_FP64, kernel)):
        flow = FlowConfig(mach=0.5, cfl=1.0, precision=prec, scheme=_lib.SCHEME_AUSM)
        state = perturbed_state(arrays, flow, 3)
        state[key][0] = value
        out.append(residual(arrays, flow, state, k)[0, 1:])
    assert np.isnan(out[0]).any()
    assert np.isnan(out[1])[np.isnan(out[0])].all()


@pytest.mark.parametrize("kernel", DOUBLE_KERNELS)
@pytest.mark.parametrize("power", [600, -600])
def test_roe_of_densities_out_of_range(power, kernel):
    """Densities and pressures whose products overflow or vanish although their roots do not: the fluxes are
    proportional to them, so a power of two comes through, within the 2e-13 of test_gpu_fast_flux.py of the
    sizes of a cell's face terms (at most eight times the largest component here)."""
    arrays = prepared("tets")
    flow = FlowConfig(mach=0.5, cfl=1.0, precision=_lib.PREC_FP64, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 3)
    n = int(arrays["n_cells"])
    scaled = {k: v.copy() for k, v in state.items()}
    for key in ("rho", "p"):
        scaled[key][:n] *= 2.0 ** power
    inner = np.ones(n, bool)  # without the cells of farfield faces, whose ghosts keep the freestream
    inner[arrays["farfield_interior"]] = False
    want = residual(arrays, flow, state, kernel)[inner]
    got = residual(arrays, flow, scaled, kernel)[inner] * 2.0 ** -power
    assert np.max(np.abs(got - want)) <= 8 * 2e-13 * np.max(np.abs(want))


@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_FP32_FLUX])
@pytest.mark.parametrize("key,value", [("p", 0.0), ("rho", 0.0), ("p", 1e-30), ("p", np.inf), ("rho", np.inf),
                                       ("u", np.inf), ("v", -np.inf), ("p", np.nan), ("rho", np.nan), ("w", np.nan)])
@pytest.mark.parametrize("name", ["channel", "ogrid", "tets"])
def test_ghosts_of_cells_out_of_range(name, key, value, precision):
    """Ghosts of cells with a zero, vanishing, infinite or undefined entry, of every boundary kind: NaN and
    infinite where the exact mode's are, and the same numbers elsewhere (30 roundings, as above)."""
    arrays = prepared(name)
    n = int(arrays["n_cells"])
    state = perturbed_state(arrays, FlowConfig(mach=0.5), 3)
    state[key][np.flatnonzero(np.random.default_rng(5).uniform(size=n) < 0.3)] = value
    got = []
    for prec in (_lib.PREC_FP64_EXACT, precision):
        flow = FlowConfig(mach=0.5, cfl=1.0, precision=prec, ordering=_lib.ORDER_SPATIAL)
        s = EulerSolver(arrays, flow, autotune=False)
        s.set_state(state)
        s.residual()
        got.append(s.get_state())
        s.close()
    tol = 900 * (2.0 ** -53 if precision == _lib.PREC_FP64 else 2.0 ** -24)
    for k in ("rho", "u", "v", "w", "p", "E", "H", "M"):
        want, have = got[0][k][n:], got[1][k][n:]
        assert np.array_equal(np.isnan(want), np.isnan(have)), k
        assert np.array_equal(np.isinf(want), np.isinf(have)), k
        w, h = want[np.isfinite(want)], have[np.isfinite(want)]
        assert np.max(np.abs(h - w) / (np.abs(w) + np.median(np.abs(w)))) <= tol, k


@pytest.mark.parametrize("kernel", DOUBLE_KERNELS)
@pytest.mark.parametrize("scheme", [_lib.SCHEME_ROE, _lib.SCHEME_AUSM])
@pytest.mark.parametrize("key", ["p", "rho"])
def test_symmetry_faces_of_one_negative_entry(key, scheme, kernel):
    """A negative pressure or density alone has no sound speed: NaN through a symmetry face, as in the
    exact mode."""
    arrays = cube()
    out = []
    for prec, k in ((_lib.PREC_FP64_EXACT, _lib.KERNEL_TILE), (_lib.PREC_FP64, kernel)):
        flow = FlowConfig(mach=0.5, cfl=1.0, precision=prec, scheme=scheme)
        state = perturbed_state(arrays, flow, 3)
        state[key][0] *= -1.0
        out.append(residual(arrays, flow, state, k)[0])
    assert np.isnan(out[0][1:4]).all()
    assert np.array_equal(np.isnan(out[0]), np.isnan(out[1]))
