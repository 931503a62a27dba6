"""Captured solves across engines and for batches: a replay has the bits of the solve
launched kernel by kernel with the same engine, whichever engine was captured before
it and whatever buffers the earlier calls had.
"""
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from hoexplicit import HighOrderExplicitOp, recon, workloads  # noqa: E402
from hoexplicit.batch import OperatorBatch  # noqa: E402


def _op(seed, shape, nSam, nCha, engine):
    w = workloads.small(seed=seed, shape=shape, nSam=nSam, nCha=nCha, nTerm=9, masked=True)
    return HighOrderExplicitOp(w.grid, w.kspha, w.times, engine=engine, **w.op_kwargs())


def _rand(g, *n):
    return torch.randn(*n, dtype=torch.complex64, generator=g).cuda()


def test_an_engine_switch_is_captured_anew():
    op = _op(9, (14, 9, 1), 301, 5, "tc")
    g = torch.Generator().manual_seed(3)
    kw = dict(iterations=4, lam=1e-2)
    kept, first = [], {}
    probe = _rand(g, op.nSam, op.nCha)
    for engine in ("tc", "fp32", "tc", "fp32"):
        op.set_engine(engine)
        for rep in range(3):      # the first is captured, the others replayed
            data, wt = _rand(g, op.nSam, op.nCha), _rand(g, op.nSam)
            a, sa = recon.solve(op, data, wt, use_graph=False, **kw)
            b, sb = recon.solve(op, data, wt, use_graph=True, **kw)
            assert torch.equal(a, b) and sa == sb
            kept += [data, wt, a, b]
        p, _ = recon.solve(op, probe, None, **kw)
        assert torch.equal(p, first.setdefault(engine, p))
    assert not torch.equal(first["tc"], first["fp32"])   # the engines' bits do differ
    op.close()


@pytest.mark.parametrize("engine", ["fp32", "tc"])
def test_batch_replay_takes_new_buffers(engine):
    ops = [_op(4, (14, 9, 1), 301, 5, engine), _op(5, (21, 17, 1), 523, 5, engine), _op(6, (10, 12, 1), 140, 5, engine)]
    batch = OperatorBatch(ops)
    g = torch.Generator().manual_seed(4)
    kept = []
    for iterations, lam, tol in ((3, 0.0, 0.0), (3, 1e-2, 0.0), (6, 1e-2, 0.3), (0, 0.0, 0.0)):
        kw = dict(iterations=iterations, lam=lam, rel_tol=tol)
        for rep in range(4):
            data = [_rand(g, op.nSam, op.nCha) for op in ops]
            wt = None if rep == 1 else [None if i == rep - 1 else _rand(g, op.nSam) for i, op in enumerate(ops)]
            a, sa = batch.recon(data, wt, use_graph=False, **kw)
            out = [torch.full((op.ncol,), float("nan"), dtype=torch.complex64, device="cuda") for op in ops]
            b, sb = batch.recon(data, wt, use_graph=True, out=out, **kw)
            assert all(torch.equal(x, y) for x, y in zip(a, b)) and sa == sb
            assert all(x is y for x, y in zip(b, out))
            if rep == 2:          # a member's own solve in between uses the same buffers
                recon.solve(ops[1], data[1], None, **kw)
            kept += [data, wt, a, b]
    batch.close()
    for op in ops:
        op.close()
