"""A solver that a batch hands back without having stepped it: what adding it queued on the batch's
stream (its control block, the wall Cp, its state moved to the first buffer after an odd run) is done by
then.  The batch's stream is the caller's and busy, so that the queued work is late."""
import numpy as np
import pytest

from cases import CASES, STATE_KEYS, perturbed_state, prepared
from euler3d_b200 import _lib
from euler3d_b200.batch import Batch
from euler3d_b200.solver import EulerSolver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("how", ["retire", "remove", "close_batch"])
@pytest.mark.parametrize("precision", [_lib.PREC_FP64, _lib.PREC_FP32_FLUX])
def test_never_stepped(precision, how):
    import torch

    arrays = prepared("ogrid")
    flow = CASES["ogrid"].flow(precision=precision, ordering=_lib.ORDER_SPATIAL)
    state = perturbed_state(arrays, flow, 3)
    alone, member = (EulerSolver(arrays, flow, autotune=False) for _ in range(2))
    for s in (alone, member):
        s.set_state(state)
        s.run(3)
    stream = torch.cuda.Stream()
    batch = Batch(stream=stream.cuda_stream)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)  # about 50 ms
    batch.add(member, max_iter=0 if how == "retire" else 5)
    if how == "retire":
        (r, stats, status), = batch.retire()
        assert r is member and status == _lib.E3D_OK and stats["iterations"] == 0
    elif how == "remove":
        assert batch.remove(member)["iterations"] == 0
    else:
        batch.close()
    got, want = member.get_state(), alone.get_state()
    for k in STATE_KEYS:
        assert np.array_equal(got[k], want[k]), k
    a, b = member.run(4), alone.run(4)
    assert a["iterations"] == b["iterations"] == 4
    assert np.array_equal(member.rms_history(), alone.rms_history())
    got, want = member.get_state(), alone.get_state()
    for k in STATE_KEYS:
        assert np.array_equal(got[k], want[k]), k
    batch.close()
    member.close()
    alone.close()


def test_destroyed_as_a_member():
    """A member's solver destroyed while its work is queued: the batch goes on with the others."""
    import torch

    arrays = prepared("tets")
    flow = CASES["tets"].flow(precision=_lib.PREC_FP64, ordering=_lib.ORDER_SPATIAL)
    stream = torch.cuda.Stream()
    batch = Batch(stream=stream.cuda_stream)
    gone, stays, alone = (EulerSolver(arrays, flow, autotune=False) for _ in range(3))
    for s in (gone, stays, alone):
        s.run(1)
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)
    for s in (gone, stays):
        batch.add(s, max_iter=6)
    batch._members.pop(gone._h.value)
    gone.close()
    assert [r for r, _, _ in batch.run_all()] == [stays]
    alone.run(6)
    got, want = stays.get_state(), alone.get_state()
    for k in STATE_KEYS:
        assert np.array_equal(got[k], want[k]), k
    batch.close()
