"""A context outlives the handles made through it, whatever the order in which
Python lets go of them."""
import gc
import weakref

import numpy as np
import pytest

import inti_b200 as inti

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", ["context", "operator"])
def test_context_collected_in_one_cycle_with_its_handles(first):
    """Everything in one reference cycle (as an exception's traceback makes
    one): the handles are given back before the context."""
    gc.collect()
    order = []

    class Box:
        pass

    box = Box()
    c = inti.Context(0)
    c._fin.detach()  # the real call comes last, whatever the order seen
    handle, destroy = c.handle, c.lib.inti_ctx_destroy
    weakref.finalize(c, order.append, "context")
    q = inti.ellipsoid_quadrature(3, 5)
    S, D = inti.single_double_layer(op=inti.Laplace(dim=3), target=q, source=q, correction={"method": "dim"}, ctx=c)
    A = inti.CombinedFieldOperator(D, S, 1.0, 0.5)
    B = inti.BatchOperator(inti.Laplace(dim=3), [q], "DL", None, ctx=c)
    assert np.isfinite(A @ np.ones(len(q))).all()
    for name, obj in (("quadrature", q), ("correction", S.correction), ("operator", S), ("combined", A), ("batch", B)):
        weakref.finalize(obj, order.append, name)
    box.all = [c, S, D, A, B, q] if first == "context" else [q, B, A, D, S, c]
    box.me = box
    del box, c, q, S, D, A, B, obj
    for _ in range(3):
        gc.collect()
    try:
        assert len(order) == 6 and order[-1] == "context", order
    finally:
        destroy(handle)
