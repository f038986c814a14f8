"""Timed cases of the operator framework: what a boundary-integral program
asks of it, through the public entry points, over the range of sizes it is
used at.

A case is a dict of plain values.  ``path`` says which call it is:

* ``apply``      one product with a corrected Nystrom operator on its own
                 surface (``GpuOperator``: device pointers, or host arrays
                 with ``host``; the transpose with ``transpose``);
* ``columns``    the same operator on a block of densities;
* ``potential``  a layer potential at points off the surface and, with
                 ``gradient``, the cotangents of density, nodes, normals and
                 weights for a given cotangent of the values;
* ``correction`` the density-interpolation correction of a surface;
* ``solve``      a whole GMRES solve of a boundary-integral equation;
* ``batch``      many surfaces and right-hand sides at once;
* ``batch_solve`` a whole batched GMRES solve.

Geometry sizes: ``kite`` has 5 nodes on each of ``size`` panels, ``sphere``
48*size^2 nodes (quadratic triangles, six-point rule), ``ellipsoid`` and the
stars 54*size^2 nodes (cube-sphere cells, 3x3 Gauss rule).
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "inti.jl_b200"))

import inti_b200 as inti  # noqa: E402

# flops of one ordered pair, FMA = 2, special functions not counted
PAIR_FLOPS = {
    ("laplace", 2): {"SL": 6, "DL": 10, "ADL": 10, "HS": 16},
    ("laplace", 3): {"SL": 11, "DL": 18, "ADL": 18, "HS": 26},
    ("helmholtz", 3): {"SL": 24, "DL": 34, "ADL": 34, "HS": 60},
}


# ----------------------------------------------------------------------------
# the cases
# ----------------------------------------------------------------------------
def _apply(name, pde, shape, size, kernel, k=0.0, precision="fp64", transpose=False, host=False):
    return {"name": name, "path": "apply", "pde": pde, "shape": shape, "size": size, "kernel": kernel, "k": k,
            "precision": precision, "transpose": transpose, "host": host}


def listed():
    return [
        # the smallest call: a planar problem of a thousand nodes inside an iterative solver
        _apply("kite_dl_1k", "laplace", "kite", 200, "DL"),
        # a fine planar curve with the kernel of Neumann problems
        _apply("kite_hs_9k", "laplace", "kite", 1801, "HS"),
        # an ordinary scattering surface while a model is being set up
        _apply("sphere_sl_3k", "helmholtz", "sphere", 8, "SL", k=5.0),
        # the transpose from host arrays: the reverse pass of a program that keeps numpy vectors
        _apply("sphere_dl_11k_transpose_host", "helmholtz", "sphere", 15, "DL", k=5.0, transpose=True, host=True),
        # the large scattering surface: 62,208 nodes at ten wavelengths per 2 pi
        _apply("sphere_sl_62k", "helmholtz", "sphere", 36, "SL", k=10.0),
        # the inner operator of a mixed-precision solve at 200,934 nodes
        _apply("ellipsoid_dl_201k_fp32c", "laplace", "ellipsoid", 61, "DL", precision="fp32c"),
        # a block of densities on one surface: many incident fields or a block method
        {"name": "sphere_dl_14k_64columns", "path": "columns", "pde": "helmholtz", "shape": "sphere", "size": 17,
         "kernel": "DL", "k": 5.0, "columns": 64},
        # shape optimisation: field values at 4,096 points and the gradient back to the surface
        {"name": "potential_gradient_52k", "path": "potential", "pde": "laplace", "size": 31, "kernel": "DL",
         "k": 0.0, "targets": 4096, "gradient": True},
        # set-up of a corrected operator on a new surface
        {"name": "sphere_correction_43k", "path": "correction", "pde": "helmholtz", "size": 30, "k": 8.0,
         "derivative": False},
        # a whole scattering solve on an ordinary surface, mixed precision
        {"name": "sphere_cfie_solve_7k", "path": "solve", "pde": "helmholtz", "shape": "sphere", "size": 12, "k": 5.0,
         "mode": "mixed"},
        # scattering by many bodies of uneven size, 64 incident waves, full precision
        {"name": "stars_8_fp64", "path": "batch", "surfaces": 8, "smallest": 7, "largest": 20, "k": 5.0, "columns": 64,
         "precision": "fp64"},
        # the whole batched solve: tensor-core inner iterations, full-precision residuals
        {"name": "stars_4_solve", "path": "batch_solve", "surfaces": 4, "smallest": 5, "largest": 12, "k": 5.0,
         "columns": 64, "mode": "mixed"},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["apply", "apply", "apply", "columns", "potential", "correction", "solve", "batch",
                       "batch_solve"])
    k = round(rng.uniform(1.0, 10.0), 3)
    if path in ("apply", "columns"):
        pde = rng.choice(["laplace", "helmholtz"])
        shape = "sphere" if pde == "helmholtz" else rng.choice(["kite", "ellipsoid"])
        if path == "columns":
            shape = "sphere" if pde == "helmholtz" else "ellipsoid"
        kernel = rng.choice(["SL", "DL", "ADL", "HS"])
        k = k if pde == "helmholtz" else 0.0
        if path == "columns":
            return {"path": path, "pde": pde, "shape": shape, "size": _log_int(rng, 5, 17), "kernel": kernel, "k": k,
                    "columns": rng.randint(2, 64)}
        lo, hi = {"kite": (40, 4000), "sphere": (4, 36), "ellipsoid": (4, 40)}[shape]
        transpose = rng.random() < 0.25  # from host arrays, as the transpose takes them
        c = _apply("", pde, shape, _log_int(rng, lo, hi), kernel, k, rng.choice(["fp64", "fp64", "fp64", "fp32c"]),
                   transpose, transpose or rng.random() < 0.25)
        del c["name"]
        return c
    if path == "potential":
        pde = rng.choice(["laplace", "helmholtz"])
        return {"path": path, "pde": pde, "size": _log_int(rng, 6, 31), "kernel": rng.choice(["SL", "DL"]),
                "k": k if pde == "helmholtz" else 0.0, "targets": _log_int(rng, 100, 4096),
                "gradient": pde == "laplace" and rng.random() < 0.7}
    if path == "correction":
        pde = rng.choice(["laplace", "helmholtz"])
        return {"path": path, "pde": pde, "size": _log_int(rng, 5, 30), "k": k if pde == "helmholtz" else 0.0,
                "derivative": rng.random() < 0.4}
    if path == "solve":
        shape = rng.choice(["kite", "sphere", "ellipsoid"])
        lo, hi = {"kite": (40, 800), "sphere": (4, 12), "ellipsoid": (4, 11)}[shape]
        pde = "helmholtz" if shape == "sphere" else "laplace"
        return {"path": path, "pde": pde, "shape": shape, "size": _log_int(rng, lo, hi),
                "k": k if pde == "helmholtz" else 0.0, "mode": "fp64" if shape == "kite" else rng.choice(["fp64", "mixed"])}
    if path == "batch":
        small = rng.randint(5, 10)
        return {"path": path, "surfaces": rng.randint(2, 8), "smallest": small, "largest": small + rng.randint(0, 10),
                "k": round(rng.uniform(1.0, 5.0), 3), "columns": rng.choice([1, 5, 16, 33, 64, 64]),
                "precision": rng.choice(["fp64", "fp64", "tf32"])}
    small = rng.randint(4, 8)
    return {"path": path, "surfaces": rng.randint(2, 4), "smallest": small, "largest": small + rng.randint(0, 4),
            "k": round(rng.uniform(1.0, 5.0), 3), "columns": rng.choice([4, 16, 64]),
            "mode": rng.choice(["fp64", "mixed"])}


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
def _op(case, dim=3):
    return inti.Helmholtz(k=case["k"], dim=3) if case.get("pde", "helmholtz") == "helmholtz" else inti.Laplace(dim=dim)


def _quadrature(shape, size):
    if shape == "kite":
        return inti.kite_quadrature(size, 9)
    return inti.p2_sphere_quadrature(size) if shape == "sphere" else inti.ellipsoid_quadrature(size, 5)


def _stars(case, seed):
    rng = np.random.default_rng(seed)
    sizes = np.linspace(case["smallest"], case["largest"], case["surfaces"]).round().astype(int)
    return [inti.star_quadrature(inti.star_coefficients(rng), int(n)) for n in sizes]


def _field(pde, k, x, seed, columns=1, radius=3.0):
    """Smooth densities at the points ``x``: fields of eight point sources
    with seeded places and strengths, ``(columns, n)``."""
    rng = np.random.default_rng(seed)
    dim = x.shape[1]
    out = np.empty((columns, len(x)), np.complex128 if pde == "helmholtz" else np.float64)
    for c in range(columns):
        s = rng.standard_normal((8, dim))
        s *= radius / np.linalg.norm(s, axis=1, keepdims=True)
        q = rng.standard_normal(8)
        d = np.linalg.norm(x[:, None, :] - s[None, :, :], axis=2)
        if pde == "helmholtz":
            out[c] = (np.exp(1j * k * d) / d) @ (q + 1j * rng.standard_normal(8))
        else:
            out[c] = (np.log(d) if dim == 2 else 1.0 / d) @ q
    return out


def _waves(k, x, seed, columns):
    """Plane waves with seeded directions at ``x``, ``(columns, n)``."""
    v = np.random.default_rng(seed).standard_normal((columns, 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return np.exp(1j * k * (v @ x.T))


def _targets(case, seed):
    """Points on the ellipsoid's 1.5-fold copy, seeded directions."""
    v = np.random.default_rng(seed + 1000).standard_normal((case["targets"], 3))
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    return 1.5 * v * np.array([1.0, 0.7, 0.5])


def _layer(case, q):
    kernel = case["kernel"]
    pair = inti.single_double_layer(op=_op(case, q.dim), target=q, source=q,
                                    compression={"method": "b200", "precision": case.get("precision", "fp64")},
                                    correction={"method": "dim"}, derivative=kernel in ("ADL", "HS"))
    return pair[0] if kernel in ("SL", "ADL") else pair[1]


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _equation(case, q):
    """The boundary-integral equation's operator: interior Dirichlet on the
    kite, the exterior combined field elsewhere."""
    S, D = inti.single_double_layer(op=_op(case, q.dim), target=q, source=q, correction={"method": "dim"})
    if q.dim == 2:
        return -0.5 * inti.I + D
    return 0.5 * inti.I + D + (-1j * case["k"]) * S if case["pde"] == "helmholtz" else 0.5 * inti.I + D + S


def prepare(case, seed):
    path = case["path"]
    st = {"case": case}
    if path in ("apply", "columns"):
        q = _quadrature(case["shape"], case["size"])
        st["op"] = _layer(case, q)
        x = _field(case["pde"], case["k"], q.coords, seed, case.get("columns", 1))
        if path == "apply" and case["host"]:
            st["x"] = x[0].copy()
        else:
            st["x"] = _cuda(x if path == "columns" else x[0])
            st["y"] = torch.zeros_like(st["x"])
    elif path == "potential":
        q = inti.ellipsoid_quadrature(case["size"], 5)
        kernel = inti.DoubleLayerKernel if case["kernel"] == "DL" else inti.SingleLayerKernel
        st["op"] = inti.IntegralOperator(kernel(_op(case)), inti.points(_targets(case, seed)), q)
        st["x"] = _cuda(_field(case["pde"], case["k"], q.coords, seed)[0])
        st["u"] = torch.zeros(case["targets"], dtype=st["x"].dtype, device="cuda")
        if case["gradient"]:
            st["g"] = _cuda(np.random.default_rng(seed + 7).standard_normal(case["targets"]))
            n = len(q)
            st["d"] = {"sigma": torch.zeros(n, device="cuda", dtype=torch.float64),
                       "coords": torch.zeros(n, 3, device="cuda", dtype=torch.float64),
                       "normals": torch.zeros(n, 3, device="cuda", dtype=torch.float64),
                       "weights": torch.zeros(n, device="cuda", dtype=torch.float64)}
    elif path == "correction":
        # a sphere whose radius the seed sets: another surface, as well conditioned
        st["q"] = inti.p2_sphere_quadrature(case["size"], 1.0 + 0.1 * np.random.default_rng(seed).random())
        st["op"] = _op(case)
    elif path == "solve":
        q = _quadrature(case["shape"], case["size"])
        st["L"] = _equation(case, q)
        st["b"] = _field(case["pde"], case["k"], q.coords, seed, radius=3.0 if q.dim == 2 else 0.2)[0]
    else:
        quads = _stars(case, seed)
        op = inti.Helmholtz(k=case["k"], dim=3)
        corr = [inti.bdim_correction(op, q, q) for q in quads]
        st["op"] = inti.BatchOperator(op, quads, "CF", corr, c_dl=1.0, c_sl=-1j * case["k"])
        x = _waves(case["k"], np.concatenate([q.coords for q in quads]), seed, case["columns"])
        if path == "batch":
            st["x"] = _cuda(x)
            st["y"] = torch.zeros_like(st["x"])
        else:
            st["b"] = np.asfortranarray(-x.T)
    return st


# ----------------------------------------------------------------------------
# one pass
# ----------------------------------------------------------------------------
def run(st):
    case = st["case"]
    path = case["path"]
    if path == "apply":
        if case["transpose"]:
            return st["op"].rmatvec(st["x"])
        if case["host"]:
            return st["op"] @ st["x"]
        st["op"].apply_device(st["x"].data_ptr(), st["y"].data_ptr())
        return st["y"]
    if path == "columns":
        st["op"].apply_device(st["x"].data_ptr(), st["y"].data_ptr(), case["columns"])
        return st["y"]
    if path == "potential":
        st["op"].apply_device(st["x"].data_ptr(), st["u"].data_ptr())
        if not case["gradient"]:
            return st["u"]
        d = st["d"]
        st["op"].grad_sources_device(st["g"].data_ptr(), st["x"].data_ptr(), d["sigma"].data_ptr(),
                                     d["coords"].data_ptr(), d["normals"].data_ptr(), d["weights"].data_ptr())
        return {"u": st["u"], "d": d}
    if path == "correction":
        dS, dD = inti.bdim_correction(st["op"], st["q"], st["q"], derivative=case["derivative"])
        rowptr, col, s = dS.arrays()
        return {"rowptr": rowptr, "col": col, "S": s, "D": dD.arrays()[2]}
    if path == "solve":
        return inti.gmres(st["L"], st["b"], rtol=1e-10, mode=case["mode"])[0]
    if path == "batch":
        st["op"].apply_device(st["x"].data_ptr(), st["y"].data_ptr(), case["columns"], case["precision"])
        return st["y"]
    return st["op"].gmres(st["b"], shift=0.5, rtol=1e-10, mode=case["mode"])[0]


# ----------------------------------------------------------------------------
# what one pass cannot do without
# ----------------------------------------------------------------------------
def _nodes(case):
    return {"kite": 5 * case["size"], "sphere": 48 * case["size"] ** 2, "ellipsoid": 54 * case["size"] ** 2}[
        case["shape"]]


def _product(pde, dim, kernel, pairs, n, columns, nq, m=None):
    """Bytes and flops of one product: nodes, densities, correction rows and
    results once; one kernel value per pair, its products per column."""
    m = n if m is None else m
    s = 16 if pde == "helmholtz" else 8
    flops = PAIR_FLOPS[(pde, dim)][kernel] * pairs + (columns - 1) * pairs * (8 if pde == "helmholtz" else 2)
    return {"bytes": 8 * n * (2 * dim + 1) + columns * s * (n + m) + n * nq * (s + 4), "flops": flops}


def work(case):
    path = case["path"]
    if path in ("apply", "columns"):
        n, dim = _nodes(case), 2 if case["shape"] == "kite" else 3
        nq = {"kite": 5, "sphere": 6, "ellipsoid": 9}[case["shape"]]
        return _product(case["pde"], dim, case["kernel"], float(n) * n, n, case.get("columns", 1), nq)
    if path == "potential":
        n, m = 54 * case["size"] ** 2, case["targets"]
        w = _product(case["pde"], 3, case["kernel"], float(n) * m, n, 1, 0, m)
        if case["gradient"]:
            w = {"bytes": w["bytes"] + 8 * (9 * n + 4 * m), "flops": w["flops"] + 40.0 * n * m}
        return w
    if path == "correction":
        n, cplx = 48 * case["size"] ** 2, case["pde"] == "helmholtz"
        f = PAIR_FLOPS[(case["pde"], 3)]["HS" if case["derivative"] else "DL"]
        return {"bytes": 8 * 7 * n + n * 6 * (2 * (16 if cplx else 8) + 4),
                "flops": float(n) * n * (f + 18 * 2 * (8 if cplx else 2))}
    if path == "solve":
        # a residual and a few Krylov products of the combined field at the least
        n, dim = _nodes(case), 2 if case["shape"] == "kite" else 3
        w = _product(case["pde"], dim, "DL", float(n) * n, n, 1, 5)
        return {"bytes": 8 * w["bytes"], "flops": 8 * w["flops"]}
    sizes = [54 * int(v) ** 2 for v in np.linspace(case["smallest"], case["largest"], case["surfaces"]).round()]
    w = [_product("helmholtz", 3, "DL", float(n) * n, n, case["columns"], 9) for n in sizes]
    times = 8 if path == "batch_solve" else 1
    return {key: times * sum(v[key] for v in w) for key in ("bytes", "flops")}


# ----------------------------------------------------------------------------
# the same values in plain 64-bit torch
# ----------------------------------------------------------------------------
def _kernel(pde, kind, k, x, nx, y, ny):
    """Kernel values K(x_i, y_j) without the weights, zero for coincident points."""
    dim = x.shape[1]
    r = [x[:, c, None] - y[None, :, c] for c in range(dim)]
    d2 = sum(a * a for a in r)
    same = d2 <= 1e-28
    d2 = torch.where(same, 1.0, d2)
    d = d2.sqrt()
    dots = {}
    if kind in ("ADL", "HS"):
        dots["x"] = sum(a * nx[:, c, None] for c, a in enumerate(r))
    if kind in ("DL", "HS"):
        dots["y"] = sum(a * ny[None, :, c] for c, a in enumerate(r))
    if kind == "HS":
        dots["n"] = nx @ ny.T
    if pde == "helmholtz":
        e = torch.polar(1 / (4 * math.pi * d), k * d)
        f = torch.complex(1 / d, torch.full_like(d, -k)) / d
        if kind == "SL":
            v = e
        elif kind == "DL":
            v = e * f * dots["y"]
        elif kind == "ADL":
            v = -e * f * dots["x"]
        else:
            g = torch.complex(k * k * d2 - 3, 3 * k * d) / (d2 * d2)
            v = e * (f * dots["n"] + g * dots["x"] * dots["y"])
    elif dim == 2:
        c = 1 / (2 * math.pi)
        if kind == "SL":
            v = -c * d.log()
        elif kind == "DL":
            v = c * dots["y"] / d2
        elif kind == "ADL":
            v = -c * dots["x"] / d2
        else:
            v = c * (dots["n"] - 2 * dots["x"] * dots["y"] / d2) / d2
    else:
        c = 1 / (4 * math.pi)
        if kind == "SL":
            v = c / d
        elif kind == "DL":
            v = c * dots["y"] / (d2 * d)
        elif kind == "ADL":
            v = -c * dots["x"] / (d2 * d)
        else:
            v = c * (dots["n"] - 3 * dots["x"] * dots["y"] / d2) / (d2 * d)
    return torch.where(same, torch.zeros((), dtype=v.dtype, device=v.device), v)


def _tensors(q):
    return _cuda(q.coords), None if q.normals is None else _cuda(q.normals), _cuda(q.weights)


def _chunks(m, n):
    step = max(1, (1 << 25) // n)
    return [slice(a, min(m, a + step)) for a in range(0, m, step)]


def _dim(pde, k, q, derivative):
    """Density-interpolation weights (dS, dD), each ``(elements, nq, nq)``:
    rows are an element's nodes, columns the same nodes."""
    x, nx, w = _tensors(q)
    n, dim = x.shape
    ns = 3 * q.nq
    lo, hi = q.coords.min(0), q.coords.max(0)
    radius = 1.5 * np.linalg.norm(hi - lo) / 2
    i = np.arange(ns)
    if dim == 2:
        s = np.stack([np.cos(2 * np.pi * i / ns), np.sin(2 * np.pi * i / ns)], 1)
    else:
        t = 1 - 2 * i / (ns - 1)
        a = np.pi * (3 - np.sqrt(5.0)) * (i + 1)
        s = np.stack([np.cos(a) * np.sqrt(1 - t * t), t, np.sin(a) * np.sqrt(1 - t * t)], 1)
    s = _cuda(radius * s + (lo + hi) / 2)
    g0, g1 = _kernel(pde, "SL", k, x, nx, s, None), _kernel(pde, "ADL", k, x, nx, s, None)
    ks, kd = ("ADL", "HS") if derivative else ("SL", "DL")
    theta = -0.5 * (g1 if derivative else g0)
    wg0, wg1 = w[:, None] * g0, w[:, None] * g1
    for c in _chunks(n, n):
        theta[c] += _kernel(pde, ks, k, x[c], nx[c], x, nx) @ wg1 - _kernel(pde, kd, k, x[c], nx[c], x, nx) @ wg0
    el = lambda v: v.reshape(-1, q.nq, ns)  # noqa: E731
    Q, R = torch.linalg.qr(torch.cat([el(g0), el(g1)], 1).transpose(1, 2))
    W = torch.linalg.solve_triangular(R, Q.mH @ el(theta).transpose(1, 2), upper=True).transpose(1, 2)
    return -W[:, :, q.nq:], W[:, :, : q.nq]


def _corrected(pde, kind, k, q, v, transpose=False, weights=None):
    """(A + C) v or its transpose, v ``(n, columns)`` on the device."""
    x, nx, w = _tensors(q)
    n = len(q)
    if weights is None:
        weights = _dim(pde, k, q, kind in ("ADL", "HS"))[0 if kind in ("SL", "ADL") else 1]
    out = torch.empty_like(v)
    back = {"SL": "SL", "DL": "ADL", "ADL": "DL", "HS": "HS"}[kind]
    for c in _chunks(n, n):
        if transpose:
            out[c] = w[c, None] * (_kernel(pde, back, k, x[c], nx[c], x, nx) @ v)
        else:
            out[c] = _kernel(pde, kind, k, x[c], nx[c], x, nx) @ (w[:, None] * v)
    e = v.reshape(-1, q.nq, v.shape[1])
    return out + ((weights.transpose(1, 2) if transpose else weights) @ e).reshape(out.shape)


def _dense(pde, k, q, terms, shift):
    """shift*I + sum of c*(A + C) as a dense matrix."""
    x, nx, w = _tensors(q)
    n = len(q)
    dS, dD = _dim(pde, k, q, False)
    A = torch.zeros(n, n, dtype=dS.dtype, device="cuda")
    block = torch.arange(n, device="cuda").reshape(-1, q.nq)
    for kind, c in terms:
        for rows in _chunks(n, n):
            A[rows] += c * _kernel(pde, kind, k, x[rows], nx[rows], x, nx) * w
        A[block[:, :, None], block[:, None, :]] += c * (dS if kind == "SL" else dD)
    A.diagonal().add_(shift)
    return A


def _split(quads):
    off = np.cumsum([0] + [len(q) for q in quads])
    return [slice(int(a), int(b)) for a, b in zip(off[:-1], off[1:])]


def exact(case, seed):
    path, k = case["path"], case["k"]
    pde = case.get("pde", "helmholtz")
    if path in ("apply", "columns"):
        q = _quadrature(case["shape"], case["size"])
        x = _cuda(_field(pde, k, q.coords, seed, case.get("columns", 1)).T)
        y = _corrected(pde, case["kernel"], k, q, x, case.get("transpose", False))
        return y[:, 0] if path == "apply" else y.T.contiguous()
    if path == "potential":
        q = inti.ellipsoid_quadrature(case["size"], 5)
        t = _cuda(_targets(case, seed))
        y, ny, w = _tensors(q)
        s = _cuda(_field(pde, k, q.coords, seed)[0])
        if not case["gradient"]:
            return torch.cat([_kernel(pde, case["kernel"], k, t[c], None, y, ny) @ (w * s)
                              for c in _chunks(len(t), len(q))])
        g = _cuda(np.random.default_rng(seed + 7).standard_normal(case["targets"]))
        leaves = [v.requires_grad_() for v in (s, y, ny, w)]
        u = []
        for c in _chunks(len(t), 4 * len(q)):
            uc = _kernel(pde, case["kernel"], k, t[c], None, y, ny) @ (w * s)
            (uc @ g[c]).backward()
            u.append(uc.detach())
        d = [torch.zeros_like(v) if v.grad is None else v.grad for v in leaves]
        return {"u": torch.cat(u), "d": dict(zip(("sigma", "coords", "normals", "weights"), d))}
    if path == "correction":
        q = inti.p2_sphere_quadrature(case["size"], 1.0 + 0.1 * np.random.default_rng(seed).random())
        dS, dD = _dim(pde, k, q, case["derivative"])
        return {"rowptr": None, "col": None, "S": dS.reshape(-1), "D": dD.reshape(-1)}
    if path == "solve":
        q = _quadrature(case["shape"], case["size"])
        b = _cuda(_field(pde, k, q.coords, seed, radius=3.0 if q.dim == 2 else 0.2)[0])
        terms = [("DL", 1.0)] if q.dim == 2 else [("DL", 1.0), ("SL", -1j * k if pde == "helmholtz" else 1.0)]
        return torch.linalg.solve(_dense(pde, k, q, terms, -0.5 if q.dim == 2 else 0.5), b)
    quads = _stars(case, seed)
    x = _cuda(_waves(k, np.concatenate([q.coords for q in quads]), seed, case["columns"]).T)
    if path == "batch":
        out = []
        for q, c in zip(quads, _split(quads)):
            dS, dD = _dim(pde, k, q, False)
            out.append(_corrected(pde, "DL", k, q, x[c], weights=dD)
                       - 1j * k * _corrected(pde, "SL", k, q, x[c], weights=dS))
        return torch.cat(out).T.contiguous()
    return torch.cat([torch.linalg.solve(_dense(pde, k, q, [("DL", 1.0), ("SL", -1j * k)], 0.5), -x[c])
                      for q, c in zip(quads, _split(quads))])
