"""Entry-wise accuracy of multi-column FP64 products whose magnitudes vary
within a row of the operator or within a density: refined surfaces, targets
close to a surface, unit vectors, narrow Gaussians, densities on one part of
a surface.

The reference is the sum in extended precision (64-bit significands) of the
kernel at the nodes' FP64 coordinates.  An entry's allowance is

    (4 m + 64 + 4 k d) eps sum_j S_ij |w_j x_j|,   eps = 2^-52,

m nonzero densities, S the modulus that the kernel's evaluation works with
(|n| d for |r.n|: the products in r.n are rounded at that size).  The parts:
rounding of a kernel value and of w x, under 32 operations of eps/2 each,
doubled; the phase k d (relative rounding of d and of the product, and the
table's, under 4 eps k d); the sum of m complex products in any order, at
most 2 m real ones, each rounded at eps/2 of the sum of moduli, twice for
m complex densities whose parts are summed apart.
"""
import numpy as np
import pytest
import torch

import inti_b200 as inti

pytestmark = pytest.mark.gpu

KERNEL = {"SL": inti.SingleLayerKernel, "DL": inti.DoubleLayerKernel, "ADL": inti.AdjointDoubleLayerKernel,
          "HS": inti.HyperSingularKernel}
LD = np.longdouble
EPS = 2.0**-52


def graded_sphere(levels=12, cells=5):
    """The unit sphere as six patches of cells x cells (odd), the middle cell of
    one refined towards its centre by `levels` halvings, 3 x 3 Gauss nodes."""
    g, w = np.polynomial.legendre.leggauss(3)
    h = 2.0 / cells
    rect = []
    for face in range(6):
        for i in range(cells):
            for j in range(cells):
                if face == 0 and i == j == cells // 2:
                    continue
                rect.append((face, -1 + i * h, -1 + j * h, h))
    s = h
    for _ in range(levels):  # the square (-s/2, s/2)^2 without its middle ninth: eight cells
        for i in range(3):
            for j in range(3):
                if not i == j == 1:
                    rect.append((0, -s / 2 + i * s / 3, -s / 2 + j * s / 3, s / 3))
        s /= 3
    rect.append((0, -s / 2, -s / 2, s))
    X, W = [], []
    for face, u0, v0, c in rect:
        u, v = np.meshgrid(u0 + c * (g + 1) / 2, v0 + c * (g + 1) / 2, indexing="ij")
        u, v, ww = u.ravel(), v.ravel(), (np.outer(w, w) * c * c / 4).ravel()
        p = np.stack([np.ones(9), np.tan(np.pi / 4 * u), np.tan(np.pi / 4 * v)], 1)
        r = np.linalg.norm(p, axis=1)
        jac = (np.pi / 4) ** 2 * (p[:, 1] ** 2 + 1) * (p[:, 2] ** 2 + 1) / r**3
        p /= r[:, None]
        sign = 1 if face < 3 else -1
        X.append(sign * np.roll(p, face % 3, axis=1))
        W.append(ww * jac)
    X = np.concatenate(X)
    return inti.Quadrature(X, X.copy(), np.concatenate(W), 9)


def reference(pde, kind, k, tgt, rows, src, X):
    """(K w X)[rows] in extended precision, and sum S |w x|."""
    x, y = tgt.coords[rows].astype(LD), src.coords.astype(LD)
    ny = src.normals.astype(LD)
    b = src.weights.astype(LD)[:, None] * X.astype(np.clongdouble if pde == "helmholtz" else LD)
    r = x[:, None, :] - y[None]
    d2 = (r * r).sum(-1)
    same = d2 <= LD(1e-28)
    d = np.sqrt(np.where(same, LD(1), d2))
    one = LD(1)
    nx = tgt.normals[rows].astype(LD) if tgt.normals is not None else None
    rny = (r * ny[None]).sum(-1)
    lnx = np.sqrt((nx * nx).sum(-1))[:, None] if nx is not None else None
    lny = np.sqrt((ny * ny).sum(-1))[None]
    f = one / d + k  # |1/d - ik| at most
    if kind == "SL":
        v, S = one / d, one / d
    elif kind == "DL":
        v, S = rny / d**2 * (one / d - 1j * LD(k) if k else one / d), f / d * lny
    else:
        rnx = (r * nx[:, None]).sum(-1)
        if kind == "ADL":
            v, S = -rnx / d**2 * (one / d - 1j * LD(k) if k else one / d), f / d * lnx
        else:
            nn = (nx[:, None] * ny[None]).sum(-1)
            kd = LD(k) * d
            v = nn / d**2 * (one / d - 1j * LD(k) if k else one / d)
            v = v + ((kd * kd - 3 + 3j * kd) if k else -3 * one) * rnx * rny / d**5
            S = (f / d**2 + (kd * kd + 3 * kd + 3) / d**3) * lnx * lny
    if pde == "helmholtz":
        v = v * (np.cos(LD(k) * d) + 1j * np.sin(LD(k) * d))
    c = one / (4 * LD(np.pi).__class__("3.14159265358979323846264338327950288"))
    v, S = np.where(same, 0, v) * c, np.where(same, 0, S) * c
    return v @ b, S @ abs(b), float(d.max())


def check(A, pde, kind, k, tgt, src, X, rows):
    Y = A @ X
    ref, T, dmax = reference(pde, kind, k, tgt, rows, src, X)
    m = (X != 0).sum(0)[None, :]
    allow = (4.0 * m + 64 + 4 * k * dmax) * EPS * T
    err = np.abs(Y[rows] - ref)
    assert (err <= allow).all(), float((err / np.maximum(allow, LD(1e-300))).max())
    return Y


def waves(q, n, cplx, seed):
    v = np.random.default_rng(seed).standard_normal((n, 3))
    p = q.coords @ v.T
    return np.exp(1j * p) if cplx else np.cos(p + 0.3)


def columns(q, family, cplx, seed=1):
    """(n, 8) densities of a family."""
    r = np.random.default_rng(seed)
    n = len(q)
    W = waves(q, 8, cplx, seed)
    if family == "smooth":
        return W
    if family == "unit":
        X = np.zeros_like(W)
        X[np.concatenate([[n - 1, n - 5], r.choice(n, 6, replace=False)]), np.arange(8)] = 1.0
        return X
    c = np.concatenate([[n - 1], r.choice(n, 7, replace=False)])
    d2 = ((q.coords[:, None] - q.coords[None, c]) ** 2).sum(-1)
    if family == "gauss":
        return np.exp(-d2 / (2 * 0.05**2)) * W
    X = W.copy()  # "part": only farther than 0.5 from a node
    X[d2 < 0.25] = 0.0
    return X


def operator(pde, kind, k, tgt, src, ctx):
    return inti.GpuOperator(KERNEL[kind](inti.Helmholtz(k=k, dim=3) if k else inti.Laplace(dim=3)), tgt, src, None,
                            "fp64", ctx)


@pytest.mark.parametrize("pde,k", [("laplace", 0.0), ("helmholtz", 4.0)])
@pytest.mark.parametrize("kind", ["SL", "DL", "ADL", "HS"])
@pytest.mark.parametrize("shape", ["graded", "uniform"])
def test_on_a_surface(ctx, pde, k, kind, shape):
    q = graded_sphere() if shape == "graded" else inti.p2_sphere_quadrature(7)
    n = len(q)
    assert n * n >= 2e6
    A = operator(pde, kind, k, q, q, ctx)
    rows = np.unique(np.concatenate([np.arange(0, n, 97), np.arange(n - 20, n)]))
    for family in ("smooth", "unit", "gauss", "part"):
        check(A, pde, kind, k, q, q, columns(q, family, bool(k)), rows)


@pytest.mark.parametrize("pde,k", [("laplace", 0.0), ("helmholtz", 4.0)])
@pytest.mark.parametrize("kind", ["DL", "HS"])
@pytest.mark.parametrize("off", [1e-3, 1e-6])
def test_close_to_a_surface(ctx, pde, k, kind, off):
    """Targets at a small distance from nodes, among targets farther away."""
    q = inti.p2_sphere_quadrature(7)
    d = np.random.default_rng(5).standard_normal((900, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    t = np.concatenate([q.coords[::50] * (1 + off), 1.5 * d])
    tgt = inti.Quadrature(t, t / np.linalg.norm(t, axis=1, keepdims=True), np.ones(len(t)), 0)
    A = operator(pde, kind, k, tgt, q, ctx)
    rows = np.concatenate([np.arange(0, 48, 3), np.arange(100, 900, 80)])
    for family in ("smooth", "unit", "gauss", "part"):
        check(A, pde, kind, k, tgt, q, columns(q, family, bool(k)), rows)


@pytest.mark.parametrize("pde,k", [("laplace", 0.0), ("helmholtz", 4.0)])
@pytest.mark.parametrize("nrhs", [8, 37])
def test_sources_taken_apart(ctx, pde, k, nrhs):
    """The hypersingular kernel's nearest sources where they are not the 40 of
    a smooth surface: 300 nodes of ordinary weight within 0.02 (more than a
    target keeps), 60 on one point, weights of zero and below it."""
    q = inti.p2_sphere_quadrature(7)
    r = np.random.default_rng(8)
    y = np.concatenate([q.coords, q.coords[100] + 0.02 * r.random((300, 3)), np.repeat(q.coords[900:901], 60, axis=0)])
    w = np.concatenate([q.weights, np.full(360, q.weights.mean())])
    w[200:260] = 0.0
    w[300:360] *= -1.0
    src = inti.Quadrature(y, y / np.linalg.norm(y, axis=1, keepdims=True), w, 0)
    A = operator(pde, "HS", k, src, src, ctx)
    rows = np.concatenate([np.arange(90, 110), np.arange(195, 365, 10), [900, 901, 2000], np.arange(2352, 2652, 30), [2700]])
    X = np.tile(columns(src, "smooth", bool(k)), (1, 5))[:, :nrhs]
    check(A, pde, "HS", k, src, src, X, rows)
    check(A, pde, "HS", k, src, src, columns(src, "unit", bool(k)), rows)


def _captured(A, X, c, s):
    """The product in a captured graph, which keeps the FP64 MMA kernel."""
    x = torch.from_numpy(X.T.copy()).cuda()
    assert x.shape[1] == A.shape[1]
    y = torch.zeros((x.shape[0], A.shape[0]), dtype=x.dtype, device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        A.apply_device(x.data_ptr(), y.data_ptr(), X.shape[1])
    g.replay()
    torch.cuda.synchronize()
    out = y.cpu().numpy().T
    del g
    return out


@pytest.mark.parametrize("pde,k", [("laplace", 0.0), ("helmholtz", 4.0)])
@pytest.mark.parametrize("kind", ["SL", "DL", "ADL", "HS"])
def test_which_form_takes_a_density(pde, k, kind):
    """Smooth densities keep the fixed-point form (other last bits than the
    FP64 MMA kernel), unit vectors and an otherwise smooth block with one
    unit vector get the FP64 MMA kernel's own bits."""
    s = torch.cuda.Stream()
    c = inti.Context(0, stream=s.cuda_stream)
    q = inti.p2_sphere_quadrature(7)
    A = operator(pde, kind, k, q, q, c)
    smooth, unit = columns(q, "smooth", bool(k)), columns(q, "unit", bool(k))
    mixed = smooth.copy()
    mixed[:, 5] = unit[:, 2]
    assert not np.array_equal(A @ smooth, _captured(A, smooth, c, s))
    for X in (unit, mixed):
        assert np.array_equal(A @ X, _captured(A, X, c, s))


@pytest.mark.parametrize("kind,n,apart", [("SL", 512, True), ("SL", 1024, False), ("HS", 1024, True), ("HS", 1728, False)])
def test_few_sources_keep_the_fp64_kernel(ctx, kind, n, apart):
    """8,000 targets: with few sources the FP64 MMA kernel is the faster form
    (its bits), with more the contraction."""
    s = torch.cuda.Stream()
    c = inti.Context(0, stream=s.cuda_stream)
    full = inti.p2_sphere_quadrature(6)
    pick = np.linspace(0, len(full) - 1, n).astype(int)
    q = inti.Quadrature(full.coords[pick], full.normals[pick], full.weights[pick], 0)
    d = np.random.default_rng(4).standard_normal((8000, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    A = operator("laplace", kind, 0.0, inti.Quadrature(1.4 * d, d, np.ones(8000), 0), q, c)
    X = columns(q, "smooth", False)
    assert np.array_equal(A @ X, _captured(A, X, c, s)) == apart


def _scale(top):
    """The power of two that takes top to (1.9, 3.8) 2^61: the splitting's unit is its inverse."""
    m, e = np.frexp(top)
    return 2.0 ** ((61 if 2 * m > 1.9 else 62) - (e - 1))


@pytest.mark.parametrize("near,heavy", [(64, 64), (1024, 8), (8, 1024)])
def test_no_digit_product_is_missing(ctx, near, heavy):
    """1,534 equal terms, so that the digits of the products add up: sources on
    a sphere about the first target, one of them `near` times closer and one of
    `heavy` times the weight, which set the scales.  Each of the eight lowest
    products that are kept is worth 9e-15 of the sum or more in one of the three
    cases (8.8e-15 the least, computed from the digits in exact arithmetic).
    Allowed: what is dropped and rounded, 2^65.2 units of the two scales per
    term, and four roundings of a term, twice: 5.2e-15 to 6.4e-15 of the sum."""
    n = 1536
    r = np.random.default_rng(3)
    d = r.standard_normal((n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    y, w = 1.5 * d, np.full(n, 1.0 / 3.0)
    y[9] /= near
    w[700] *= heavy
    src = inti.Quadrature(y, d, w, 0)
    far = r.standard_normal((1400, 3))
    far *= 4.0 / np.linalg.norm(far, axis=1, keepdims=True)
    tgt = inti.points(np.concatenate([np.zeros((1, 3)), far]))
    A = operator("laplace", "SL", 0.0, tgt, src, ctx)
    X = np.ones((n, 8)) * 2.0 ** np.arange(8)
    Y = A @ X
    ref, T, _ = reference("laplace", "SL", 0.0, tgt, np.arange(1), src, X)
    K = 1.0 / np.linalg.norm(y, axis=1)
    units = _scale(K.max()) * np.array([_scale(w.max() * c) for c in 2.0 ** np.arange(8)])
    allow = n * 2.0**65.2 / units / (4 * np.pi) + 8 * 2.0**-53 * T[0]
    assert (allow <= 7e-15 * T[0]).all()
    assert (np.abs(Y[0] - ref[0]) <= allow).all(), np.abs(Y[0] - ref[0]) / T[0]


@pytest.mark.parametrize("pde,k", [("laplace", 0.0), ("helmholtz", 4.0)])
@pytest.mark.parametrize("derivative", [False, True])
def test_theta_of_a_refined_surface(ctx, pde, k, derivative):
    """The density interpolation of targets on a refined surface: with one
    target more the product is large enough for the fixed-point form.  Its
    kernel values and traces do not fit it, so every other row keeps the FP64
    kernel's bits (rows are summed apart, in chunks that depend on the number
    of 128-row blocks only); on a uniform surface the rows change theirs."""
    limit = {(False, False): 5e7, (False, True): 2e7, (True, False): 8.8e7, (True, True): 3.3e7}[derivative, bool(k)]
    op = inti.Helmholtz(k=k, dim=3) if k else inti.Laplace(dim=3)
    cells, nsub = {5e7: (13, 14), 2e7: (9, 10), 8.8e7: (13, 15), 3.3e7: (11, 12)}[limit]
    for q, same in ((graded_sphere(12, cells), True), (inti.p2_sphere_quadrature(nsub), False)):
        n = len(q)
        m = int(np.ceil(limit / n)) - 1
        assert m < n and (m + 127) // 128 == (m + 128) // 128
        pick = np.random.default_rng(2).permutation(n)
        pick = np.concatenate([np.arange(n - 30, n), pick[pick < n - 30]])  # the refined corner first
        rows = []
        for count in (m, m + 1):
            t = inti.Quadrature(q.coords[pick[:count]], q.normals[pick[:count]], np.ones(count), 0)
            dS, dD = inti.bdim_correction(op, t, q, green_multiplier=-0.5, derivative=derivative, ctx=ctx)
            rows.append([c.arrays()[2][: m * q.nq] for c in (dS, dD)])
        equal = all(np.array_equal(a, b) for a, b in zip(*rows))
        assert equal == same
