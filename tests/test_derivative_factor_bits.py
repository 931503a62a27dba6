"""The derivative product's factor is no less accurate than in FP32.

The phase is zero here and the image nonzero only at voxels where the factor
F[s,v] = sum_l kdot[l,s] bf[v,l] vanishes for every sample, while its terms do not:
what the product returns there is the error of F, and nothing of the later BF16
split.  Basis and coefficients are FP32 values, so the oracle's FP64 value has no
input rounding in it.

Tolerance: the error, over all samples, of the same reduced factor evaluated in
FP32 as written down below (tables rounded to FP32, one FMA a term), on the same
problem.
"""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

from hoexplicit import Grid, HighOrderExplicitOp  # noqa: E402
from hoexplicit.model import basisfunc_spha  # noqa: E402
from tests.test_gpu_parity import host, maybe_skip  # noqa: E402

f32 = lambda a: np.asarray(a, np.float64).astype(np.float32)  # noqa: E731


def _fma(a, b, c):
    """FP32 FMA: the product is exact in FP64."""
    return f32(a.astype(np.float64) * b + c)


def _factor_fp32(bf, kdot):
    """2 pi F [samples, voxels of bf's first rows given] in FP32 from the reduced basis."""
    g = bf.T @ bf
    d = np.zeros(len(g))
    d[np.diag(g) > 0] = 1 / np.sqrt(np.diag(g)[np.diag(g) > 0])
    w, v = np.linalg.eigh(g * d[:, None] * d)
    v = v[:, w > 1e-9 * w.max()]
    tab = f32(bf @ (d[:, None] * v))
    M = f32(np.where(d[:, None] > 0, v / np.where(d > 0, d, 1)[:, None], 0))
    kd = np.zeros((kdot.shape[1], v.shape[1]), np.float32)
    for l in range(len(g)):
        kd = _fma(f32(kdot[l])[:, None], M[l][None], kd)
    kd = f32(kd.astype(np.float64) * np.float32(2 * np.pi))
    return tab, kd


@pytest.mark.parametrize("shape,nTerm", [((29, 18, 1), 9), ((29, 18, 1), 16), ((13, 10, 6), 9), ((13, 10, 6), 16)])
@pytest.mark.parametrize("nCha", [1, 16])
def test_factor_is_as_accurate_as_fp32(shape, nTerm, nCha):
    maybe_skip("tc")
    nSam = 4096
    rng = np.random.default_rng(nTerm + shape[2])
    d = 2.0 ** -7
    grid = Grid(*shape, d, d, d)
    bf = basisfunc_spha(grid.x, grid.y, grid.z, list(range(1, nTerm + 1)))
    assert np.array_equal(bf, f32(bf))
    n = len(bf)
    norm = np.linalg.norm(bf, axis=0)
    norm[norm == 0] = 1
    zero = rng.choice(n, 4, replace=False)            # where F vanishes
    B = bf[zero] / norm
    kdot = rng.standard_normal((nTerm, nSam))
    kdot = f32((kdot - np.linalg.pinv(B) @ (B @ kdot)) / norm[:, None]).astype(np.float64)
    x = np.zeros(n, np.complex64)
    x[zero] = [1, -1, 1, 1]
    exact = 2j * np.pi * (kdot.T @ (bf.T @ x.astype(np.complex128))) / np.sqrt(n)
    op = HighOrderExplicitOp(grid, np.zeros((nTerm, nSam)), np.arange(nSam) * 2e-6, engine="tc", kspha_dt=kdot,
                             csm=np.ones(shape + (nCha,), np.complex128))
    y = host(op * torch.from_numpy(x).cuda()).reshape(nCha, nSam)
    op.close()
    err = np.sqrt(np.mean(np.abs(y - exact) ** 2))
    tab, kd = _factor_fp32(bf, kdot)
    F = np.zeros((nSam, 4), np.float32)
    for k in range(kd.shape[1]):
        F = _fma(kd[:, k][:, None], tab[zero, k][None], F)
    tol = np.sqrt(np.mean(np.abs(1j * (F.astype(np.float64) @ x[zero].real) / np.sqrt(n) - exact) ** 2))
    print(f"{shape} {nTerm} {nCha}: {err / tol:.3f} of FP32's error {tol:.3e}")
    assert err <= tol
