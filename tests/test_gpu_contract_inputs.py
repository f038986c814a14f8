"""Inputs of multi-column products (8 columns and more, 2e6 pairs and more)
that the fixed-point contraction has to take, or hand over to the FP64
kernels, as those always did."""
import numpy as np
import pytest
import torch

import inti_b200 as inti
from helpers import density

pytestmark = pytest.mark.gpu


def _points(n, seed):
    r = np.random.default_rng(seed)
    d = r.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    return inti.Quadrature(d * np.array([1.0, 0.7, 0.5]), d, r.random(n) / n, 0)


def test_more_columns_than_a_grid_dimension_holds(ctx):
    """65,544 columns (a grid's second dimension ends at 65,535) that repeat
    eight densities: every repetition gives the eight columns' values, up to
    the rounding of the last addition (1e-13 leaves n eps of 1,440 sources)."""
    n, nrhs = 1440, 65544
    q = _points(n, 1)
    A = inti.GpuOperator(inti.SingleLayerKernel(inti.Laplace(dim=3)), q, q, None, "fp64", ctx)
    X = np.stack([density(n, False, c) for c in range(8)], axis=1)
    ref = torch.from_numpy((A @ X).T.copy()).cuda()
    x = torch.from_numpy(X.T.copy()).cuda().repeat(nrhs // 8, 1)
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    A.apply_device(x.data_ptr(), y.data_ptr(), nrhs)
    ctx.synchronize()
    d = y.view(nrhs // 8, 8, n).sub_(ref)
    assert (d.norm(dim=2).amax(0) <= 1e-13 * ref.norm(dim=1)).all()


@pytest.mark.parametrize("pde", ["laplace", "helmholtz"])
@pytest.mark.parametrize("coefs", [(np.nan, 1.0), (1.0, np.nan), (np.inf, 1.0)])
def test_coefficients_that_are_not_finite(ctx, pde, coefs):
    """A combined field with such a coefficient: no entry of the block of
    columns is finite, as in products of one column."""
    cplx = pde == "helmholtz"
    op = inti.Helmholtz(k=3.0, dim=3) if cplx else inti.Laplace(dim=3)
    q = _points(1500, 2)
    S = inti.GpuOperator(inti.SingleLayerKernel(op), q, q, None, "fp64", ctx)
    D = inti.GpuOperator(inti.DoubleLayerKernel(op), q, q, None, "fp64", ctx)
    A = inti.CombinedFieldOperator(D, S, *coefs)
    X = np.stack([density(1500, cplx, c) for c in range(9)], axis=1)
    assert not np.isfinite(A @ X[:, 0]).any()
    assert not np.isfinite(A @ X).any()
