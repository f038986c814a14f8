"""Multi-column products of more than 2e6 pairs and the Theta product of
large corrections: the contraction on the INT8 tensor path (contract_i8.cu).

Sizes are taken at its edges: a last row block of one target and of 128, a
last source stage of one source (stages hold 64 real or 32 complex sources),
column widths on both sides of a multiple of eight and of a pass (32 complex,
64 real columns).  The reference is the oracle's FP64 row sums.  Both sides
carry the rounding of the kernel values (a few 1e-16) and the oracle that of
its n-term sums (at most n * 1.1e-16 * sum|K x| / |sum K x|, a few 1e-13 at
n = 2,000 for these densities), so 1e-12 holds for either form.
"""
import numpy as np
import pytest

import inti_b200 as inti
import oracle as O
from helpers import density, relerr

pytestmark = pytest.mark.gpu

KERNEL = {"SL": inti.SingleLayerKernel, "DL": inti.DoubleLayerKernel, "ADL": inti.AdjointDoubleLayerKernel,
          "HS": inti.HyperSingularKernel}
OKIND = {"SL": O.SL, "DL": O.DL, "ADL": O.ADL, "HS": O.HS}


def _points(n, seed, scale=1.0):
    """n points and unit normals of an ellipsoid-like surface, no element structure."""
    r = np.random.default_rng(seed)
    d = r.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return inti.Quadrature(scale * d * np.array([1.0, 0.7, 0.5]), d, r.random(n) / n, 0)


def _columns(n, nrhs, cplx, seed):
    return np.stack([density(n, cplx, seed + c) for c in range(nrhs)], axis=1)


@pytest.mark.parametrize("pde", ["laplace", "helmholtz"])
@pytest.mark.parametrize("kind", ["SL", "DL", "ADL", "HS"])
@pytest.mark.parametrize("m,n,nrhs", [(1537, 1473, 8), (1536, 1409, 33), (1665, 1505, 65), (129, 20001, 17)])
def test_contraction_matches_oracle(ctx, pde, kind, m, n, nrhs):
    cplx = pde == "helmholtz"
    op = inti.Helmholtz(k=6.0, dim=3) if cplx else inti.Laplace(dim=3)
    src, tgt = _points(n, 1), _points(m, 2, 1.3)
    A = inti.GpuOperator(KERNEL[kind](op), tgt, src, None, "fp64", ctx)
    X = _columns(n, nrhs, cplx, 5)
    Y = A @ X
    for c in {0, nrhs // 2, nrhs - 1}:
        ref = O.apply(O.HELMHOLTZ if cplx else O.LAPLACE, OKIND[kind], 6.0 if cplx else 0.0, tgt.coords, tgt.normals,
                      src.coords, src.normals, src.weights, X[:, c])
        assert relerr(Y[:, c], ref) < 1e-12


@pytest.mark.parametrize("pde", ["laplace", "helmholtz"])
def test_contraction_on_the_surface_with_correction_and_beta(ctx, pde):
    """Self pairs, correction rows, alpha and beta, padded leading dimensions."""
    import torch

    cplx = pde == "helmholtz"
    op = inti.Helmholtz(k=3.0, dim=3) if cplx else inti.Laplace(dim=3)
    q = inti.ellipsoid_quadrature(6, 5)  # 1,944 nodes
    S, D = inti.single_double_layer(op=op, target=q, source=q, correction={"method": "dim"}, ctx=ctx)
    A = inti.CombinedFieldOperator(D, S, 1.0, -3.0j if cplx else 0.4)
    n, nrhs, ld = len(q), 19, len(q) + 5
    X, Y0 = _columns(ld, nrhs, cplx, 1), _columns(ld, nrhs, cplx, 100)
    alpha, beta = (0.5 - 0.25j, 0.75 + 0.1j) if cplx else (0.5, 0.75)
    x = torch.from_numpy(X.T.copy()).cuda()
    y = torch.from_numpy(Y0.T.copy()).cuda()
    torch.cuda.synchronize()
    A.apply_device(x.data_ptr(), y.data_ptr(), nrhs, alpha, beta, ldx=ld, ldy=ld)
    ctx.synchronize()
    got = y.cpu().numpy().T
    ref = np.stack([A @ X[:n, c] for c in range(nrhs)], axis=1)  # single products, checked against the oracle
    assert relerr(got[:n], alpha * ref + beta * Y0[:n]) < 1e-12
    assert np.array_equal(got[n:], Y0[n:])


def test_contraction_is_independent_of_column_scales(ctx):
    """Each column has its own power-of-two scale: columns of size 1e100 and
    1e-100 and a zero column next to ordinary ones are as accurate as these."""
    q = _points(1600, 3)
    A = inti.GpuOperator(inti.SingleLayerKernel(inti.Laplace(dim=3)), q, q, None, "fp64", ctx)
    X = _columns(1600, 12, False, 9)
    X[:, 4] = 0.0
    f = np.ones(12)
    f[[2, 7]] = 2.0**330, 2.0**-330
    Y, Z = A @ X, A @ (X * f)
    assert np.array_equal(Z, Y * f)
    assert not Y[:, 4].any()


@pytest.mark.parametrize("bad", [np.inf, np.nan, 1e300])
def test_contraction_hands_over_densities_out_of_range(ctx, bad):
    """Columns that do not fit the fixed-point form go to the FP64 kernels:
    the other columns are exact, the bad one as in single products."""
    q = _points(1600, 4)
    A = inti.GpuOperator(inti.SingleLayerKernel(inti.Laplace(dim=3)), q, q, None, "fp64", ctx)
    X = _columns(1600, 9, False, 2)
    X[700, 5] = bad
    Y = A @ X
    ref = np.stack([A @ X[:, c] for c in range(9)], axis=1)
    keep = [c for c in range(9) if c != 5]
    assert relerr(Y[:, keep], ref[:, keep]) < 1e-12
    assert np.array_equal(np.isfinite(Y[:, 5]), np.isfinite(ref[:, 5]))
    if np.isfinite(bad):
        assert relerr(Y[:, 5] / bad, ref[:, 5] / bad) < 1e-12  # (norms of 1e295 overflow)


def test_captured_product_runs_without_the_shared_buffers(ctx):
    """A product captured into a graph keeps the FP64 MMA kernel, whose
    launches name no buffer of the context: replays after a larger product
    (which replaces those buffers) are the same."""
    import torch

    s = torch.cuda.Stream()
    c = inti.Context(0, stream=s.cuda_stream)
    op = inti.Laplace(dim=3)
    q, big = _points(1500, 5), _points(3000, 6)
    A = inti.GpuOperator(inti.DoubleLayerKernel(op), q, q, None, "fp64", c)
    x = torch.from_numpy(_columns(1500, 10, False, 1).T.copy()).cuda()
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        A.apply_device(x.data_ptr(), y.data_ptr(), 10)
    g.replay()
    torch.cuda.synchronize()
    first = y.clone()
    B = inti.GpuOperator(inti.DoubleLayerKernel(op), big, big, None, "fp64", c)
    B @ _columns(3000, 64, False, 3)
    y.zero_()
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(first, y)
    assert relerr(first.cpu().numpy().T, A @ x.cpu().numpy().T) < 1e-12
    del g


@pytest.mark.parametrize("pde,nsub", [("laplace", 13), ("helmholtz", 10)])
@pytest.mark.parametrize("derivative", [False, True])
def test_theta_of_large_corrections_matches_oracle(ctx, pde, nsub, derivative):
    """Corrections whose Theta takes the contraction (8,112 and 4,800 nodes):
    weights of sampled elements within the bound of test_gpu_dim.py."""
    from helpers import dim_values_close, oracle_dim_csr

    q = inti.p2_sphere_quadrature(nsub)
    k = 5.0 if pde == "helmholtz" else 0.0
    op = inti.Helmholtz(k=k, dim=3) if k else inti.Laplace(dim=3)
    opde = O.HELMHOLTZ if k else O.LAPLACE
    got = inti.bdim_correction(op, q, q, derivative=derivative, ctx=ctx)
    els = np.random.default_rng(1).choice(q.nel, 24, replace=False)
    els.sort()
    ref = oracle_dim_csr(opde, k, q, derivative=derivative, elements=els)
    for g, r in zip(got, ref):
        assert dim_values_close(opde, k, q, g.arrays(), r, elements=els) <= 1.0
