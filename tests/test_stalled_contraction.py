"""The contraction's instances leave a wait that runs out as one warp: the
operands of one stage of CTA 0 are not fetched (HOE_INJECT_TC_STALL, waits of 1 ms,
once), the call reports the timeout, and the next products are those of an
operator without the injection, bit for bit.  Coil widths of 8, 16, 32 and 64 (with
32 there are more phase-warp groups than units in the ring) and a stage of the first
pair, which is loaded before the kernel before has ended, or a later one.
"""
import os

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from hoexplicit import HighOrderExplicitOp, HoeError, workloads  # noqa: E402
from hoexplicit import _lib as L  # noqa: E402
from tests.test_gpu_parity import dev, maybe_skip  # noqa: E402


@pytest.mark.parametrize("nCha", [4, 16, 32, 64])
@pytest.mark.parametrize("stage", [0, 7])
def test_stall(nCha, stage):
    maybe_skip("tc")
    w = workloads.small(seed=12, shape=(64, 64, 1), nSam=4000, nCha=nCha, nTerm=16)   # some 13 stages per CTA
    make = lambda: HighOrderExplicitOp(w.grid, w.kspha, w.times, engine="tc", **w.op_kwargs())  # noqa: E731
    ref = make()
    os.environ["HOE_INJECT_TC_STALL"] = str(stage)
    try:
        op = make()
    finally:
        del os.environ["HOE_INJECT_TC_STALL"]
    x = dev(w.x)
    op * x
    with pytest.raises(HoeError) as exc:
        op.check()
    assert f"[{L.HOE_ERR_TIMEOUT}]" in str(exc.value)
    want = ref * x
    assert torch.equal(op * x, want)
    assert torch.equal(op.H * want, ref.H * want)
    op.check()
    ref.close()
    op.close()
