"""One-sided FP64 products at the edges of their launch shapes: target counts
around the 64 and 128 rows of a block, source counts around the 32- and
128-source units, few and many chunks, corrections and alpha/beta, against
the oracle.  A product of n sources differs from the oracle's by the order of
its FP64 sums: at most about n eps of the sum of magnitudes (3e-12 at the
13,000 sources here, and near sqrt(n) eps in practice), taken as 1e-12 of the
norm as for every FP64 product."""
import numpy as np
import pytest
import torch

import inti_b200 as inti
import oracle as O
from helpers import density, oracle_apply, relerr

pytestmark = pytest.mark.gpu

KERNELS = {"SL": (inti.SingleLayerKernel, O.SL), "DL": (inti.DoubleLayerKernel, O.DL),
           "ADL": (inti.AdjointDoubleLayerKernel, O.ADL), "HS": (inti.HyperSingularKernel, O.HS)}


@pytest.fixture(scope="module")
def tiled():
    c = inti.Context(0)
    c.set_single_launch(False)
    return c


def _points(n, dim, seed):
    r = np.random.default_rng(seed)
    X, N = r.standard_normal((n, dim)), r.standard_normal((n, dim))
    N /= np.linalg.norm(N, axis=1, keepdims=True)
    return inti.Quadrature(X, N, r.uniform(0.5, 1.5, n), 0)


@pytest.mark.parametrize("case", ["laplace2d", "laplace3d", "helmholtz3d"])
@pytest.mark.parametrize("m,n", [(1, 1), (1, 33), (63, 128), (64, 129), (65, 4097), (129, 31), (300, 13001),
                                 (2049, 1500), (4100, 6100)])
def test_launch_shapes(tiled, case, m, n):
    dim = 2 if case == "laplace2d" else 3
    src, tgt = _points(n, dim, 7 + m), _points(m, dim, 9 + n)
    op = inti.Helmholtz(k=3.0, dim=3) if case == "helmholtz3d" else inti.Laplace(dim=dim)
    pde, k = (O.HELMHOLTZ, 3.0) if case == "helmholtz3d" else (O.LAPLACE, 0.0)
    cplx = pde == O.HELMHOLTZ
    x, y0 = density(n, cplx, 6), density(m, cplx, 8)
    rng = np.random.default_rng(11)
    per = min(3, n)
    rp = np.arange(0, per * m + 1, per, dtype=np.int64)
    col = np.concatenate([np.sort(rng.choice(n, per, replace=False)) for _ in range(m)]).astype(np.int32)
    val = density(per * m, cplx, 12)
    alpha, beta = (0.5 - 0.25j, 1.5 + 0.5j) if cplx else (0.5, 1.5)
    rows = np.arange(m) if m < 1000 else np.arange(0, m, 17)
    for kname, (K, okind) in KERNELS.items():
        C = inti.CorrectionMatrix.from_csr(rp, col, val, (m, n), ctx=tiled)
        A = inti.GpuOperator(K(op), tgt, src, C, "fp64", tiled)
        assert not A.tuning["single_launch"]
        ref = (alpha * (oracle_apply(pde, okind, k, tgt, src, x, rows=rows) + O.csr_apply(rp, col, val, x)[rows])
               + beta * y0[rows])
        y = A.mul(y0.copy(), x, alpha=alpha, beta=beta)
        assert relerr(y[rows], ref) < 1e-12, kname
        assert np.array_equal(A.mul(y0.copy(), x, alpha=alpha, beta=beta), y)


@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("m,n", [(1, 1), (3, 65), (64, 63), (130, 64), (513, 129), (4100, 300)])
def test_source_gradients(tiled, dim, m, n):
    """Source gradients at the edges of their blocks (64 sources, 128 staged
    targets, four shares of a stage) against automatic differentiation of the
    dense product; the sums are over at most 4,100 targets."""
    src, tgt = _points(n, dim, 3 + m), inti.points(_points(m, dim, 5 + n).coords)
    g, sig = density(m, False, 2), density(n, False, 4)
    for K in (inti.SingleLayerKernel, inti.DoubleLayerKernel):
        A = inti.GpuOperator(K(inti.Laplace(dim=dim)), tgt, src, None, "fp64", tiled)
        got = A.grad_sources(g, sig)
        s, y, ny, w = (torch.tensor(np.array(v), requires_grad=True)
                       for v in (sig, src.coords, src.normals, src.weights))
        r = torch.tensor(np.array(tgt.coords))[:, None, :] - y[None]
        d2 = (r * r).sum(-1)
        if K is inti.SingleLayerKernel:
            M = -torch.log(d2) / (4 * np.pi) if dim == 2 else d2 ** -0.5 / (4 * np.pi)
        else:
            rn = (r * ny[None]).sum(-1)
            M = rn / (2 * np.pi * d2) if dim == 2 else rn * d2 ** -1.5 / (4 * np.pi)
        (torch.tensor(g) @ (M @ (w * s))).backward()
        for name, v in (("sigma", s), ("coords", y), ("normals", ny), ("weights", w)):
            want = np.zeros(tuple(v.shape)) if v.grad is None else v.grad.numpy()
            assert np.linalg.norm(got[name] - want) <= 1e-12 * np.linalg.norm(want), (K, name)
