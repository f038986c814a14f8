"""The buffers of multi-column products belong to the context while operators
use them, and go back with the last of these."""
import gc

import numpy as np
import pytest
import torch

import inti_b200 as inti

pytestmark = pytest.mark.gpu


def test_buffers_go_back_with_the_last_operator():
    """64 complex columns at 37,632 nodes take 77 MB of digit blocks (1,176
    stages of 2 x 64 x 512 bytes) and 154 MB of partial sums (1,176 slots of
    2 x 64 x 128 doubles); blocks of 64 MB and more come from the driver and go
    straight back to it.  They stay while another operator that has used them
    lives, and the products are the same after they are gone."""
    c = inti.Context(0)
    q, small = inti.p2_sphere_quadrature(28), inti.p2_sphere_quadrature(6)
    K = inti.SingleLayerKernel(inti.Helmholtz(k=2.0, dim=3))
    v = np.random.default_rng(0).standard_normal((64, 3))

    def product(op, x):
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        op.apply_device(x.data_ptr(), y.data_ptr(), 64)
        c.synchronize()
        return y

    def free():
        gc.collect()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    x, xs = (torch.from_numpy(np.exp(1j * (p.coords @ v.T)).T.copy()).cuda() for p in (q, small))
    A, B = (inti.GpuOperator(K, p, p, None, "fp64", c) for p in (q, small))
    y, ys = product(A, x), product(B, xs)
    full = free()
    del A
    assert free() - full < 100 << 20  # B may still use them
    del B
    assert free() - full >= 200 << 20
    A, B = (inti.GpuOperator(K, p, p, None, "fp64", c) for p in (q, small))
    assert torch.equal(product(A, x), y) and torch.equal(product(B, xs), ys)
