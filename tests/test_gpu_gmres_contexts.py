"""Two contexts of one device that solve at the same time, each on its own
thread: a context's lock covers its own calls only, so nothing that a solve
sets may belong to the device."""
import threading

import numpy as np
import pytest

import inti_b200 as inti
from helpers import density

pytestmark = pytest.mark.gpu


def test_small_solves_of_two_contexts_with_different_restarts(ctx):
    """Small-system cycles whose shared memory differs (restart 2 and 1,000,
    the smallest in use and the largest): every solve returns, bit for bit,
    what the same solve returns alone."""
    def problem(c):
        q = inti.ellipsoid_quadrature(4, 5)
        _, D = inti.single_double_layer(op=inti.Laplace(dim=3), target=q, source=q, correction={"method": "dim"},
                                        ctx=c)
        return D - 0.5 * inti.I, density(len(q), False, 3)

    jobs = [(inti.Context(0), 2, 240), (inti.Context(0), 1000, 60)]
    alone, errors, got = [], [], [[], []]
    for c, restart, maxiter in jobs:
        L, b = problem(c)
        alone.append((L, b, inti.gmres(L, b, rtol=1e-15, restart=restart, maxiter=maxiter)[0]))
    start = threading.Barrier(2)

    def solve(t):
        L, b, _ = alone[t]
        try:
            start.wait(30)
            for _ in range(20):
                got[t].append(inti.gmres(L, b, rtol=1e-15, restart=jobs[t][1], maxiter=jobs[t][2])[0])
        except Exception as e:  # noqa: BLE001 - reported by the assertion below
            errors.append((jobs[t][1], repr(e)))

    threads = [threading.Thread(target=solve, args=(t,)) for t in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for t in range(2):
        assert all(np.array_equal(x, alone[t][2]) for x in got[t])
