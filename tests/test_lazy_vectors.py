"""Lazily conjugated and negated tensors (x.conj(), series.conj().imag) hold other
values in memory than they read as; every entry point takes what they read as.
The expected values come from the same call on the values written out, so they
are equal bit for bit.
"""
from types import SimpleNamespace

import numpy as np
import pytest

torch = pytest.importorskip("torch")

import hoexplicit  # noqa: E402
from hoexplicit import HighOrderExplicitOp, coils, recon, workloads  # noqa: E402
from hoexplicit import sync as hsync  # noqa: E402
from hoexplicit.batch import OperatorBatch  # noqa: E402
from hoexplicit.operator import _direct, _Vec  # noqa: E402


def _lazy(v):
    """(name, lazy tensor, the same values written out)"""
    yield "conj", v.conj(), v.conj_physical()
    yield "neg", torch._neg_view(v), -v
    yield "both", torch._neg_view(v.conj()), -v.conj_physical()
    m = v.reshape(-1, 7)
    yield "matrix", m.conj(), m.conj_physical()
    yield "adjoint", m.t().contiguous().mH, m.t().contiguous().mH.resolve_conj()


def test_vectors_are_written_out():
    op = SimpleNamespace(torch_device=torch.device("cpu"), device=0)
    v = torch.randn(21, dtype=torch.complex64)
    for name, lazy, plain in _lazy(v):
        t = _Vec(op, lazy, 21, "x").t
        assert not t.is_conj() and not t.is_neg() and torch.equal(t, plain.reshape(-1)), name
        d = recon._device_vector(op, lazy.reshape(21, 1), 21, 1, "Data")
        assert not d.is_conj() and not d.is_neg() and torch.equal(d, plain.reshape(-1)), name


def _op(engine, nCha=7):
    w = workloads.small(seed=3, shape=(14, 9, 1), nSam=301, nCha=nCha, nTerm=9, masked=True)
    return w, HighOrderExplicitOp(w.grid, w.kspha, w.times, engine=engine, **w.op_kwargs())


def _rand(n, seed):
    return torch.randn(n, dtype=torch.complex64, generator=torch.Generator().manual_seed(seed)).cuda()


@pytest.mark.gpu
@pytest.mark.parametrize("engine", ["fp32", "tc"])
def test_products(engine):
    _, op = _op(engine)
    nrm = hoexplicit.normalOperator(op, np.linspace(0.5, 2, op.nrow))
    batch = OperatorBatch([op])
    x, y = _rand(op.ncol, 1), _rand(op.nrow, 2)
    new = lambda n: torch.zeros(n, dtype=torch.complex64, device="cuda")  # noqa: E731
    for f, put, v, n in ((lambda a: op * a, op.prod_, x, op.nrow), (lambda a: op.H * a, op.ctprod_, y, op.ncol),
                         (lambda a: nrm * a, nrm.prod_, x, op.ncol),
                         (lambda a: batch.forward([a])[0], None, x, op.nrow),
                         (lambda a: batch.adjoint([a])[0], None, y, op.ncol),
                         (lambda a: batch.normal([a])[0], None, x, op.ncol)):
        for name, lazy, plain in _lazy(v):
            assert not _direct(op, lazy, v.numel()), name
            want = f(plain)
            assert torch.equal(f(lazy), want), name
            assert torch.equal(f(lazy.cpu()).cpu(), want.cpu()), name
            if put is None or name == "adjoint":     # in place: contiguous operands only
                continue
            assert torch.equal(put(new(n), lazy), want), name
            for out in (new(n).conj(), torch._neg_view(new(n))):
                assert put(out, lazy) is out and torch.equal(out, want), name
    op.close()


@pytest.mark.gpu
def test_gradient_solver_coils_and_series():
    w, op = _op("tc", nCha=1)
    x, y = _rand(op.ncol, 1), _rand(op.nrow, 2)
    for _, lx, px in _lazy(x):
        for a, b in zip(op.backward(lx, y.conj()), op.backward(px, y.conj_physical())):
            assert torch.equal(a, b)
    data = y.reshape(op.nSam, 1)
    kw = dict(iterations=3, lam=1e-3)
    want, _ = recon.solve(op, data.conj_physical(), None, **kw)
    batch = OperatorBatch([op])
    for out in (None, torch.zeros_like(x), torch.zeros_like(x).conj()):
        assert torch.equal(recon.solve(op, data.conj(), None, out=out, **kw)[0], want)
        got = batch.recon([data.conj()], out=None if out is None else [out], **kw)[0][0]
        assert torch.equal(got, want)
        assert out is None or torch.equal(out, want)
    t = coils.CoilCompressionTransform(np.array([[2 + 1j]]), np.ones(1), 1.0)
    assert torch.equal(coils.apply_coil_compression(data.conj(), t),
                       coils.apply_coil_compression(data.conj_physical(), t))
    k = torch.randn(40, 9, dtype=torch.complex128, device="cuda")
    assert torch.equal(hsync.InterpTrajTime(k.conj().imag, 2e-6, 1e-6), hsync.InterpTrajTime(-k.imag, 2e-6, 1e-6))
    kt = torch._neg_view(torch.from_numpy(np.ascontiguousarray(w.kspha.T)).cuda()).t()
    hsync.set_kspha(op, kt)
    a = op * x
    hsync.set_kspha(op, kt.resolve_neg().clone())
    assert torch.equal(op * x, a)
    op.close()
