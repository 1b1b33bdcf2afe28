"""Runs on a stream that may use a part of the GPU only (a green context of eight SMs): the resident
kernel is taken where every tile fits on those SMs at once, the stage kernels otherwise, with the same
bits as on the whole GPU."""
import numpy as np
import pytest

from cases import STATE_KEYS, perturbed_state
from euler3d_b200 import _lib, meshgen as mg
from euler3d_b200.solver import EulerSolver, FlowConfig, Mesh

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def small_stream():
    cu = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) == 2 else r[1:]

    ok(cu.cuInit(0) + (None,))
    dev = ok(cu.cuDeviceGet(0))
    ok(cu.cuDevicePrimaryCtxRetain(dev))
    sms = ok(cu.cuDeviceGetDevResource(dev, cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
    groups = ok(cu.cuDevSmResourceSplitByCount(1, sms, 0, 8))[0]
    assert groups[0].sm.smCount == 8
    desc = ok(cu.cuDevResourceGenerateDesc([groups[0]], 1))
    green = ok(cu.cuGreenCtxCreate(desc, dev, cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
    stream = ok(cu.cuGreenCtxStreamCreate(green, cu.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
    yield int(stream)
    cu.cuStreamDestroy(stream)
    cu.cuGreenCtxDestroy(green)
    cu.cuDevicePrimaryCtxRelease(dev)


@pytest.mark.parametrize("precision", [_lib.PREC_FP64_EXACT, _lib.PREC_FP64, _lib.PREC_FP32_FLUX])
@pytest.mark.parametrize("size,fits", [((8, 8, 2), True), ((17, 15, 2), True), ((99, 97, 2), False)])
def test_part_of_the_gpu(small_stream, size, fits, precision):
    arrays = Mesh.from_raw(mg.bump_channel(*size)).arrays()
    flow = FlowConfig(mach=0.5, cfl=1.0, precision=precision, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 9, amp=0.02)
    out = []
    for stream in (None, small_stream):
        s = EulerSolver(arrays, flow, stream=stream, autotune=False)
        s.set_state(state)
        stats = [s.run(n) for n in (7, 40)]
        out.append((stats, s.get_state(), s.rms_history()))
        s.close()
    assert all(st["kernel_launches"] == 1 for st in out[0][0])
    assert all((st["kernel_launches"] == 1) == fits for st in out[1][0])
    assert [st["iterations"] for st in out[1][0]] == [7, 40]
    assert np.array_equal(out[0][2], out[1][2])
    for k in STATE_KEYS:
        assert np.array_equal(out[0][1][k], out[1][1][k]), k
