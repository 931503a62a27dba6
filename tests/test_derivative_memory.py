"""The derivative product's tables take the memory that the factor's rank asks for:
96 bytes a voxel and a sample up to rank 8, 128 up to 10, 192 up to 16 (three BF16
parts, six products), and 0.4 MB of fixed size.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from hoexplicit import HighOrderExplicitOp, workloads  # noqa: E402
from tests.test_gpu_parity import dev, maybe_skip  # noqa: E402


@pytest.mark.parametrize("shape,nTerm,row", [((160, 150, 1), 9, 96), ((160, 150, 1), 16, 128), ((40, 30, 20), 16, 192)])
def test_table_bytes(shape, nTerm, row):
    maybe_skip("tc")
    w = workloads.small(seed=4, shape=shape, nSam=9001, nCha=2, nTerm=nTerm, masked=False)
    op = HighOrderExplicitOp(w.grid, w.kspha, w.times, engine="tc", kspha_dt=w.kspha_dt, **w.op_kwargs())
    pad = lambda n: (n + 127) // 128 * 128  # noqa: E731
    rows = pad(int(np.prod(shape))) + pad(9001)
    before = op.info()["device_bytes"]
    for _ in range(2):
        op * dev(w.x)
        more = op.info()["device_bytes"] - before
        assert rows * row <= more <= rows * row + 400_000
    op.close()
