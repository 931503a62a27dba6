"""An operator that takes up the tensor-core engine while a replacement of its
coefficients is still queued on another stream gets the new coefficients' anchors:
the same bits as an operator that had the engine from the start.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from hoexplicit import HighOrderExplicitOp, workloads  # noqa: E402
from hoexplicit import sync as hsync  # noqa: E402
from tests.test_gpu_parity import dev, maybe_skip  # noqa: E402


@pytest.mark.parametrize("take", ["set_engine", "autotune"])
def test_engine_taken_up_behind_a_queued_replan(take):
    maybe_skip("tc")
    w = workloads.small(seed=5, shape=(23, 18, 1), nSam=700, nCha=3)
    v = workloads.small(seed=6, shape=(23, 18, 1), nSam=700, nCha=3)
    k = torch.from_numpy(np.ascontiguousarray(workloads.prepared_model(v)[1].T)).cuda().t()
    x = dev(w.x)
    ref = HighOrderExplicitOp(w.grid, w.kspha, w.times, engine="tc", **w.op_kwargs())
    hsync.set_kspha(ref, k)
    want = ref * x
    op = HighOrderExplicitOp(w.grid, w.kspha, w.times, engine="fp32", **w.op_kwargs())
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        torch.cuda._sleep(400_000_000)      # some 0.2 s of work before the replacement
        hsync.set_kspha(op, k)
    if take == "autotune":
        op.autotune(1)
    op.set_engine("tc")
    side.synchronize()
    assert torch.equal(op * x, want)
    hsync.set_kspha(op, k)                  # and once the engine is there
    assert torch.equal(op * x, want)
    ref.close()
    op.close()
