"""The anchor tables' paired FP32 arithmetic over the products that it takes, and
both tables' change to FP64 above them.

On the CPU: the kernel's steps written down in numpy, at products up to the
limit in its source, against exact sums; the error has to stay below 2^-31 cycles, a
32nd of the half ulp (2^-26) to which a table entry near 1/2 is rounded when it
is stored, so that the tables are what FP64 sums give.

On the GPU: products below and above the limit in either table against the FP64
oracle, with the engines' own tolerances (as in test_anchor_tables.py).
"""
import re
from fractions import Fraction
from pathlib import Path

import numpy as np
import pytest

SOURCE = Path(__file__).resolve().parent.parent / "highordermri.jl_gb300" / "csrc" / "hoe_anchor.cu"
f32 = lambda a: np.asarray(a, np.float64).astype(np.float32)  # noqa: E731


def _limit():
    return float(re.search(r"kPairLimit = ([0-9.]+)f", SOURCE.read_text()).group(1))


def _fma(a, b, c):
    """FP32 FMA (the product of two FP32 values is exact in FP64)."""
    return f32(a.astype(np.float64) * b + c)


def _paired(row, col):
    """frac(row . col) as k_anchor_tables forms it: [entries, components]."""
    rh, ch = f32(row), f32(col)
    rl, cl = f32(row - rh), f32(col - ch)
    hs = np.zeros(len(row), np.float32)
    ls = np.zeros(len(row), np.float32)
    add = lambda a, b: f32(a.astype(np.float64) + b)  # noqa: E731
    for l in range(row.shape[1]):
        np_ = f32(rh[:, l].astype(np.float64) * -ch[:, l])
        e = _fma(rh[:, l], ch[:, l], np_)
        e = _fma(rl[:, l], ch[:, l], _fma(rh[:, l], cl[:, l], e))
        k = add(add(np_, np.float32(12582912)), np.float32(-12582912))
        f = add(np_, -k)
        fh = add(add(f, np.float32(192)), np.float32(-192))
        hs = add(hs, fh)
        ls = add(add(ls, add(f, -fh)), -e)
    a = add(hs, -np.rint(hs))
    return -(add(a, -np.rint(add(a, ls))).astype(np.float64) + ls)


@pytest.mark.parametrize("components", [10, 17, 21])
@pytest.mark.parametrize("part", [1.0, 2.0 ** -7])
def test_paired_sums_up_to_the_limit(components, part):
    rng = np.random.default_rng(components)
    n, top = 4000, _limit() * part
    # every component's product up to the limit, split unevenly between the sides
    size = np.exp(rng.uniform(-8, 8, components))
    row = rng.uniform(-1, 1, (n, components)) * size
    col = rng.uniform(-1, 1, (n, components)) * top / size
    got = _paired(row, col)
    worst = 0.0
    for i in range(n):
        exact = sum((Fraction(a) * Fraction(b) for a, b in zip(row[i], col[i])), Fraction(0))
        d = Fraction(float(got[i])) - exact
        worst = max(worst, abs(float(d - round(d))))
    print(f"{components} components, products up to {top:g}: {worst:.2e} cycles")
    assert worst < 2.0 ** -31


@pytest.mark.gpu
@pytest.mark.parametrize("engine", ["tc", "fp32"])
@pytest.mark.parametrize("offset,ramp", [(8.0e3, 0.0), (1.0e4, 0.0), (1.9e6, 0.0), (0.0, 8.0e3), (0.0, 1.0e4),
                                         (0.0, 1.9e6), (5.0e6, 3.0e6)])
def test_large_products_in_either_table(engine, offset, ramp):
    """The constant term: its offset goes into the sample tiles' anchors (table B),
    its spread within a tile into the samples' own part (table A)."""
    pytest.importorskip("torch")
    from hoexplicit import HighOrderExplicitOp, workloads
    from hoexplicit import sync as hsync
    from oracle import dense, oracle
    from tests.test_gpu_parity import TOL, dev, host, maybe_skip
    maybe_skip(engine)
    nSam = 128 * 2 + 77
    w = workloads.small(seed=8, shape=(19, 14, 1), nSam=nSam, nCha=3, conc=True)
    w.kspha[0] += offset + ramp * np.random.default_rng(2).uniform(-1, 1, nSam)
    bf, k, t, f, c, idx = workloads.prepared_model(w)
    m = oracle.Model(bf, k, t, f, c, nTerm=16)
    y = (np.random.default_rng(3).standard_normal((2, nSam * 3)) * 0.5).astype(np.float32)
    y = (y[0] + 1j * y[1]).astype(np.complex64)
    yo, xo = oracle.forward(m, w.x[idx]), oracle.adjoint(m, y)
    op = HighOrderExplicitOp(w.grid, w.kspha, w.times, engine=engine, **w.op_kwargs())
    for again in (False, True):
        if again:
            hsync.set_kspha(op, k)
        assert dense.rel(host(op * dev(w.x)), yo) < TOL[engine]
        assert dense.rel(host(op.H * dev(y))[idx], xo) < TOL[engine]
    op.close()
