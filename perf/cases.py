"""The calls a user of this package makes, at the sizes they are made at.

An inversion builds one engine per mesh and survey and then evaluates data,
misfit and gradient for one model after another; a Gauss-Newton step
linearizes at a model and multiplies by J and J^T; the solver interface
factorizes new values on a fixed pattern and solves.  Each case below is one
such call on a new model (or new values).  The engine or solver is built once
for a mesh and survey, and its models follow one another on it, as in an
inversion.

`exact` restates the same numbers in float64 with plain torch: the nodal
finite-volume operators on a tensor mesh, a block-tridiagonal elimination over
the mesh's slabs (dense for the solver cases) and the adjoint-state gradient.
"""
from functools import lru_cache
import math

import numpy as np
import torch

DEV = "cuda"
_F64 = torch.float64


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # a first look at a line: a few thousand nodes, nothing but latency
        {"name": "dc2d_first_look_f64", "kind": "dc2d", "nx": 64, "nz": 32, "pad": 0, "nel": 15,
         "step": 3, "nsep": 4, "wenner": False, "nky": 11, "dtype": "float64"},
        # a field profile (dc2d_small's mesh and electrodes): one evaluation of an inversion
        {"name": "dc2d_profile_f64", "kind": "dc2d", "nx": 100, "nz": 50, "pad": 10, "nel": 21,
         "step": 2, "nsep": 6, "wenner": False, "nky": 11, "dtype": "float64"},
        # a long line with 96 electrodes (dc2d_large), double precision: the 2.5-D default
        {"name": "dc2d_long_line_f64", "kind": "dc2d", "nx": 400, "nz": 120, "pad": 12, "nel": 96,
         "step": 4, "nsep": 20, "wenner": True, "nky": 12, "dtype": "float64"},
        # the same line with the float32 factor and float64 refinement
        {"name": "dc2d_long_line_f32", "kind": "dc2d", "nx": 400, "nz": 120, "pad": 12, "nel": 96,
         "step": 4, "nsep": 20, "wenner": True, "nky": 12, "dtype": "float32"},
        # a small 3-D patch with an odd number of sources, float32 + refinement
        {"name": "dc3d_patch_f32", "kind": "dc3d", "nx": 33, "ny": 27, "nz": 15, "pad": 6,
         "grid": 7, "nsrc": 67, "nrx": 21, "dtype": "float32"},
        # the 3-D survey (dc3d: 269,001 nodes, 200 sources), float32 + refinement and float64
        {"name": "dc3d_survey_f32", "kind": "dc3d", "nx": 64, "ny": 64, "nz": 32, "pad": 8,
         "grid": 10, "nsrc": 200, "nrx": 30, "dtype": "float32"},
        {"name": "dc3d_survey_f64", "kind": "dc3d", "nx": 64, "ny": 64, "nz": 32, "pad": 8,
         "grid": 10, "nsrc": 200, "nrx": 30, "dtype": "float64"},
        # a Gauss-Newton step's share of the engine: linearize, then J v and J^T u per CG iteration
        {"name": "gauss_newton_line_f64", "kind": "newton", "nx": 181, "nz": 63, "pad": 9, "nel": 41,
         "step": 3, "nsep": 8, "wenner": False, "nky": 12, "iters": 4, "dtype": "float64"},
        # surveys of uneven size evaluated together
        {"name": "survey_batch_f64", "kind": "batch", "surveys": 12, "cells": 3000, "spread": 4.0,
         "nky": 12, "dtype": "float64"},
        # the regularised model-space system of a Gauss-Newton step: refactorize, one right-hand side
        {"name": "model_space_solve_f64", "kind": "solve", "mtype": "spd", "dim": 2, "nx": 150,
         "ny": 70, "nz": 1, "nbatch": 1, "nrhs": 1, "coords": False, "grad": False,
         "dtype": "float64"},
        # complex resistivity on a profile: complex-symmetric systems, data and both gradients
        {"name": "complex_resistivity", "kind": "cr", "nx": 100, "nz": 50, "pad": 10, "nel": 21,
         "step": 2, "nsep": 6, "wenner": False, "nky": 11, "dtype": "complex128"},
        # systems without symmetry through the differentiable solve, forward and backward
        {"name": "general_batch_solve_f64", "kind": "solve", "mtype": "general", "dim": 3, "nx": 19,
         "ny": 17, "nz": 13, "nbatch": 3, "nrhs": 24, "coords": True, "grad": True,
         "dtype": "float64"},
    ]


def _between(rng, lo, hi):
    """A whole number between lo and hi, spread over their logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dc2d", "dc2d", "dc3d", "dc3d", "newton", "batch", "solve", "cr"])
    real = rng.choice(["float64", "float32"])
    if kind in ("dc2d", "newton", "cr"):
        big = {"dc2d": 400, "newton": 240, "cr": 160}[kind]
        nx = _between(rng, 40, big)
        nz = max(16, int(nx * rng.uniform(0.28, 0.5)))
        step = rng.choice([1, 2, 3, 4])
        nel = max(7, min(96, int(nx * rng.uniform(0.5, 0.9)) // step))
        c = {"kind": kind, "nx": nx, "nz": nz, "pad": rng.randint(0, 12), "nel": nel, "step": step,
             "nsep": rng.randint(3, 16), "wenner": rng.random() < 0.5, "nky": rng.randint(8, 12),
             "dtype": real}
        if kind == "newton":
            c["iters"] = rng.randint(2, 5)
        if kind == "cr":
            c["dtype"] = "complex128"
        return c
    if kind == "dc3d":
        f32 = real == "float32"
        nx = _between(rng, 14, 60 if f32 else 48)
        ny = max(12, int(nx * rng.uniform(0.6, 1.0)))
        grid = max(3, min(10, (nx - 4) // 4, (ny - 4) // 2))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": max(8, int(nx * rng.uniform(0.3, 0.5))),
                "pad": rng.randint(2, 8), "grid": grid,
                "nsrc": rng.randint(1, min(200, 2 * grid * grid - 1)),
                "nrx": rng.randint(4, max(5, min(30, grid * (grid - 1)))), "dtype": real}
    if kind == "batch":
        return {"kind": kind, "surveys": rng.randint(2, 20), "cells": _between(rng, 1200, 6000),
                "spread": round(rng.uniform(1.0, 6.0), 2), "nky": rng.randint(9, 12), "dtype": real}
    mtype = rng.choice(["spd", "spd", "symmetric", "general"])
    dim = rng.choice([2, 3])
    c = {"kind": "solve", "mtype": mtype, "dim": dim}
    if dim == 2:
        c.update(nx=_between(rng, 20, 130), ny=rng.randint(17, 70), nz=1)
    else:
        c.update(nx=_between(rng, 6, 24), ny=rng.randint(6, 18), nz=rng.randint(5, 16))
    c.update(nbatch=rng.randint(1, 4), nrhs=_between(rng, 1, 70), coords=rng.random() < 0.5,
             grad=rng.random() < 0.6,
             dtype={"spd": real, "symmetric": "complex128", "general": "float64"}[mtype])
    return c


# ------------------------------------------------------- geometry (plain numpy)
def _widths(dx, n, pad, both):
    """n cells of width dx, `pad` cells growing by 1.3 outwards on the left / bottom side, and on
    the other side too with `both`."""
    g = dx * 1.3 ** np.arange(1, pad + 1)
    return np.concatenate([g[::-1], np.full(n, dx)] + ([g] if both else []))


def _geometry(c):
    """Cell widths per axis, origin, and the electrodes (node indices along the horizontal axes) of
    the sources (a, b or -1) and of the data (source, m, n)."""
    if "ny" not in c:
        h = [_widths(1.0, c["nx"], c["pad"], True), _widths(1.0, c["nz"], c["pad"], False)]
        first = c["pad"] + (c["nx"] - (c["nel"] - 1) * c["step"]) // 2
        node = first + c["step"] * np.arange(c["nel"])
        src, dat = [], []
        for i in range(c["nel"] - 2):
            mn = [(i + 1 + s, i + 2 + s) for s in range(1, c["nsep"] + 1) if i + 2 + s < c["nel"]]
            if mn:
                src.append((node[i], node[i + 1]))
                dat += [(len(src) - 1, node[m], node[n]) for m, n in mn]
        if c["wenner"]:
            for i in range(c["nel"] - 3):
                src.append((node[i], node[i + 3]))
                dat.append((len(src) - 1, node[i + 1], node[i + 2]))
        src = np.array(src)[:, :, None]
        dat_s, mn = np.array([d[0] for d in dat]), np.array([d[1:] for d in dat])[:, :, None]
        return h, src[:, 0], src[:, 1], dat_s, mn[:, 0], mn[:, 1]
    h = [_widths(5.0, c["nx"], c["pad"], True), _widths(5.0, c["ny"], c["pad"], True),
         _widths(5.0, c["nz"], c["pad"], False)]
    g = c["grid"]
    sx, sy = max(1, (c["nx"] - 4) // g), max(1, (c["ny"] - 4) // g)
    ox, oy = c["pad"] + (c["nx"] - sx * (g - 1)) // 2, c["pad"] + (c["ny"] - sy * (g - 1)) // 2
    el = np.array([(ox + sx * i, oy + sy * j) for i in range(g) for j in range(g)])
    pairs = [(i * g + j, (i + 1) * g + j) for i in range(g - 1) for j in range(g)]
    pairs += [(i * g + j, i * g + j + 1) for i in range(g) for j in range(g - 1)]
    pairs = np.array(pairs)
    sources = np.vstack([el, el + [sx // 2, sy // 2], el + [1, 0]])
    sources = sources[np.random.default_rng(7).permutation(len(sources))][:c["nsrc"]]
    at, am, an = [], [], []
    for s, e in enumerate(sources):
        far = np.linalg.norm(el[pairs].mean(1) - e, axis=1)
        far[(np.abs(el[pairs] - e).sum(-1) == 0).any(1)] = np.inf
        for p in np.argsort(far, kind="stable")[:c["nrx"]]:
            at.append(s)
            am.append(el[pairs[p, 0]])
            an.append(el[pairs[p, 1]])
    return h, sources, None, np.array(at), np.array(am), np.array(an)


def _axes(h):
    """Node coordinates: horizontal axes centred on 0, the surface at 0."""
    return [(-w.sum() if a == len(h) - 1 else -0.5 * w.sum()) + np.concatenate([[0.0], np.cumsum(w)])
            for a, w in enumerate(h)]


def _place(x, nodes):
    return np.column_stack([x[a][nodes[:, a]] for a in range(nodes.shape[1])]
                           + [np.zeros(len(nodes))])


def _wavenumbers(c):
    """(points, weights) of the inverse cosine transform: trapezoid in log k over the survey."""
    lo, hi = 0.05 / (c["nel"] * c["step"]), 6.0 / c["step"]
    k = np.exp(np.linspace(math.log(lo), math.log(hi), c["nky"]))
    w = k * math.log(hi / lo) / (c["nky"] - 1) / math.pi
    return k, w


def _half_space(c):
    """Data of a 100 ohm-m half-space with the noise floor of the survey."""
    h, a, b, at, m, n = _geometry(c)
    x = _axes(h)
    pa, pm, pn = _place(x, a)[at], _place(x, m), _place(x, n)
    inv = lambda p, q: 1.0 / np.linalg.norm(p - q, axis=1)  # noqa: E731
    d = inv(pa, pm) - inv(pa, pn)
    if b is not None:
        pb = _place(x, b)[at]
        d = d - inv(pb, pm) + inv(pb, pn)
    d = d * 100.0 / (2.0 * math.pi)
    return d, 0.05 * np.median(np.abs(d))


# -------------------------------------------------------- engines and inputs
@lru_cache(maxsize=3)
def _engine(key):
    """The engine or solver of one mesh and survey (or pattern), kept while its models follow."""
    import simpeg_dc_torch_b200 as dct
    from simpeg_dc_torch_b200 import batch, cr2d, mesh, solver, survey
    c = dict(key)
    if c["kind"] == "solve":
        crow, col, coords = _pattern(c)
        make = solver.make_solver if c["nbatch"] == 1 else solver.make_batch_solver
        size = (len(crow) - 1, c["nrhs"]) + (() if c["nbatch"] == 1 else (c["nbatch"],))
        return make(torch.as_tensor(crow), torch.as_tensor(col), *size, device=DEV,
                    dtype=getattr(torch, c["dtype"]), matrix_type=c["mtype"],
                    coords=coords if c["coords"] else None)

    def problem(c):
        h, a, b, at, m, n = _geometry(c)
        x = _axes(h)
        pa, pm, pn = _place(x, a), _place(x, m), _place(x, n)
        pb = None if b is None else _place(x, b)
        src = []
        for s in range(len(a)):
            rx = [survey.DipoleReceiver(pm[at == s], pn[at == s])]
            src.append(survey.PoleSource(rx, pa[s]) if pb is None
                       else survey.DipoleSource(rx, pa[s], pb[s]))
        return mesh.TensorMesh(h, origin=[v[0] for v in x]), survey.Survey(src)

    dt = getattr(torch, c["dtype"])
    # float32 lines are refined to the level of the float64 ones
    tol = {"refine_tol": 1e-11} if c["dtype"] == "float32" and c["kind"] != "dc3d" else {}
    if c["kind"] == "batch":
        return batch.TorchDC2DBatch([problem(p) for p in _lines(c)], nky=c["nky"], device=DEV,
                                    dtype=dt, **tol)
    if c["kind"] == "dc3d":
        return dct.TorchDC3D(*problem(c), device=DEV, dtype=dt)
    cls = cr2d.TorchCR2D if c["kind"] == "cr" else dct.TorchDC2D
    return cls(*problem(c), nky=c["nky"], device=DEV, dtype=dt, quadrature=_wavenumbers(c), **tol)


def _get_engine(c):
    return _engine(tuple(sorted((k, v) for k, v in c.items() if k != "name")))


def _lines(c):
    """The lines of a batch: sizes spread over a factor `spread`."""
    out = []
    for i in range(c["surveys"]):
        cells = c["cells"] * c["spread"] ** (((i * 5) % c["surveys"]) / max(1, c["surveys"] - 1))
        nz = max(12, int(math.sqrt(cells / 3.0)) - 6)
        nx = max(30, int(cells / (nz + 6)) - 12)
        out.append({"nx": nx + i % 2, "nz": nz, "pad": 6, "nel": 12 + (7 * i) % (nx // 2 - 11),
                    "step": 2 if i % 3 else 1, "nsep": 6, "wenner": False})
    for p in out:
        p["nel"] = min(p["nel"], (p["nx"] - 2) // p["step"])
    return out


def _model(c, rng):
    """log-resistivity on the cells: 100 ohm-m with two bodies and 10 % of cell noise."""
    h = _geometry(c)[0]
    mid = [0.5 * (v[1:] + v[:-1]) for v in _axes(h)]
    grid = np.meshgrid(*mid, indexing="ij")
    size = c["nx"] * (5.0 if "ny" in c else 1.0)
    m = math.log(100.0) + 0.1 * rng.standard_normal(grid[0].shape)
    for rho in (10.0, 1000.0):
        d2 = ((grid[-1] + size * rng.uniform(0.08, 0.2)) / (0.06 * size)) ** 2
        for g in grid[:-1]:
            d2 = d2 + ((g - size * rng.uniform(-0.25, 0.25)) / (0.1 * size)) ** 2
        m = m + math.log(rho / 100.0) * np.exp(-d2 ** 2)
    return m.reshape(-1, order="F")


def _survey_inputs(c, rng):
    """(m, dobs, w) of one line or grid: observed apparent resistivities vary around the
    half-space's, with 5 % errors and a floor."""
    d0, floor = _half_space(c)
    dobs = d0 * np.exp(0.3 * rng.standard_normal(d0.size)) + floor * rng.standard_normal(d0.size)
    return _model(c, rng), dobs, 1.0 / (0.05 * np.abs(dobs) + floor)


def _inputs(c, seed):
    """The case's inputs as float64 (complex128) numpy arrays."""
    rng = np.random.default_rng([int(seed), 17])
    if c["kind"] == "solve":
        return _solve_inputs(c, rng)
    if c["kind"] == "batch":
        parts = [_survey_inputs(p, rng) for p in _lines(c)]
        m, dobs, w = (np.concatenate(x) for x in zip(*parts))
        return {"m": m, "dobs": dobs, "w": w}
    m, dobs, w = _survey_inputs(c, rng)
    out = {"m": m, "dobs": dobs, "w": w}
    if c["kind"] == "newton":
        out["v"] = rng.standard_normal((c["iters"], m.size))
        out["u"] = rng.standard_normal((c["iters"], dobs.size)) * w
    if c["kind"] == "cr":
        out["m"] = np.concatenate([m, 0.05 * (1.0 + rng.random(m.size))])
        out["dobs"] = np.abs(dobs)
        out["dobs_ip"] = -0.07 * (1.0 + 0.2 * rng.standard_normal(dobs.size))
    return out


def _pattern(c):
    """CSR pattern of the 5-point (2-D) or 7-point (3-D) grid, and the grid coordinates."""
    shape = (c["nx"], c["ny"], c["nz"])
    idx = np.arange(c["nx"] * c["ny"] * c["nz"]).reshape(shape, order="F")
    r, q = [idx.reshape(-1)], [idx.reshape(-1)]
    for a in range(3):
        lo = np.take(idx, range(shape[a] - 1), a).reshape(-1)
        hi = np.take(idx, range(1, shape[a]), a).reshape(-1)
        r += [lo, hi]
        q += [hi, lo]
    r, q = np.concatenate(r), np.concatenate(q)
    order = np.lexsort((q, r))
    r, q = r[order], q[order]
    crow = np.concatenate([[0], np.cumsum(np.bincount(r, minlength=idx.size))])
    g = np.unravel_index(np.arange(idx.size), shape, order="F")
    coords = np.column_stack(g[:c["dim"]]).astype(np.int32)
    return crow.astype(np.int32), q.astype(np.int32), coords


def _solve_inputs(c, rng):
    """Values of diffusion systems with random coefficients (symmetric, or with a drift), b and the
    cotangent of the solution."""
    crow, col, _ = _pattern(c)
    n, nb = len(crow) - 1, c["nbatch"]
    row = np.repeat(np.arange(n), np.diff(crow))
    off = row != col
    lo, hi = np.minimum(row, col), np.maximum(row, col)
    _, pair = np.unique(lo[off].astype(np.int64) * n + hi[off], return_inverse=True)
    vals = np.zeros((nb, len(col)), np.complex128 if c["mtype"] == "symmetric" else np.float64)
    for i in range(nb):
        k = np.exp(0.8 * rng.standard_normal(pair.max() + 1))[pair]
        if c["mtype"] == "symmetric":
            k = k * (1.0 - 0.1j * rng.random(pair.max() + 1)[pair])
        if c["mtype"] == "general":
            k = k * (1.0 + 0.3 * np.sign(col[off] - row[off]))
        d = np.zeros(n, vals.dtype)
        np.add.at(d, row[off], k)
        vals[i, off] = -k
        vals[i, ~off] = d + np.exp(rng.standard_normal(n)) * 0.05
    def rhs(lead):
        x = rng.standard_normal(lead + (n, c["nrhs"]))
        return x + 1j * rng.standard_normal(x.shape) if c["mtype"] == "symmetric" else x
    lead = () if nb == 1 else (nb,)
    return {"vals": vals[0] if nb == 1 else vals, "b": rhs(()), "gx": rhs(lead)}


def prepare(case, seed):
    dt = getattr(torch, case["dtype"])
    if case["kind"] != "solve":
        dt = _F64  # models, data and weights are float64 whatever the engine's own precision
    st = {k: torch.as_tensor(v, device=DEV).to(dt) for k, v in _inputs(case, seed).items()}
    st.update(case=case, engine=_get_engine(case))
    return st


# --------------------------------------------------------------- one pass
def run(state):
    eng, c = state["engine"], state["case"]
    if c["kind"] == "solve":
        from simpeg_dc_torch_b200.solver import sparse_solve, sparse_solve_batch
        if not c["grad"]:
            eng.factorize(state["vals"])
            return {"x": eng.solve(state["b"])}
        vals = state["vals"].detach().requires_grad_(True)
        b = state["b"].detach().requires_grad_(True)
        x = (sparse_solve if c["nbatch"] == 1 else sparse_solve_batch)(vals, b, eng)
        x.backward(state["gx"])
        return {"x": x.detach(), "grad_vals": vals.grad, "grad_b": b.grad}
    if c["kind"] == "newton":
        lin = eng.linearize(state["m"])
        jv = [lin.Jvec(v) for v in state["v"]]
        jtu = [lin.Jtvec(u) for u in state["u"]]
        return {"data": lin.d, "Jv": jv, "Jtu": jtu}
    m = state["m"].detach().requires_grad_(True)
    if c["kind"] == "cr":
        d, ip = eng.dpred(m)
        phi = ((state["w"] * (d - state["dobs"])) ** 2).sum() + ((ip - state["dobs_ip"]) ** 2).sum()
        phi.backward()
        return {"data": d.detach(), "ip": ip.detach(), "phi": phi.detach(), "grad": m.grad}
    d = eng.dpred(m)
    phi = ((state["w"] * (d - state["dobs"])) ** 2).sum()
    phi.backward()
    return {"data": d.detach(), "phi": phi.detach(), "grad": m.grad}


# ------------------------------------------------------------------- work
def work(case):
    """Nested dissection of an n-node grid: about 7.75 n log2 n (2-D) or 9.4 n^(4/3) (3-D) factor
    entries and 20 n^1.5 or 5.2 n^2 operations to form them; a solve takes 4 operations per entry
    and right-hand side.  Bytes: inputs and outputs once, the factor written once and read by
    each of a solve's two sweeps, the solutions written and read once."""
    def system(n, dim):
        if dim == 2:
            return 7.75 * n * math.log2(n), 20.0 * n ** 1.5
        return 9.4 * n ** (4.0 / 3.0), 5.2 * n ** 2

    def one(nodes, cells, dim, nsys, nrhs, solves, dtype, extra):
        nnz, fac = system(nodes, dim)
        nnz = min(nnz, nodes * (nodes + 1) / 2)
        size = {"float32": 4, "float64": 8, "complex128": 16}[dtype]
        mul = 4 if dtype == "complex128" else 1
        flops = mul * nsys * (fac + 4.0 * nnz * nrhs * solves)
        by = nsys * (size * nnz * (1 + 2 * solves) + max(8, size) * 2.0 * nodes * nrhs * solves)
        return flops, by + 8.0 * (2 * cells + extra)

    def shape(c):
        h, a, _, at, _, _ = _geometry(c)
        return (np.prod([len(w) + 1 for w in h]), np.prod([len(w) for w in h]), len(h), len(a),
                len(at))

    k = case["kind"]
    if k == "solve":
        n = case["nx"] * case["ny"] * case["nz"]
        f, by = one(n, n, case["dim"], case["nbatch"], case["nrhs"], 2 if case["grad"] else 1,
                    case["dtype"], 14.0 * n)
        f *= 2 if case["mtype"] == "general" else 1
        by *= 2 if case["mtype"] == "general" else 1
        return {"bytes": by, "flops": f}
    tot = [0.0, 0.0]
    for c in (_lines(case) if k == "batch" else [case]):
        nn, nc, dim, ns, nd = shape(c)
        solves = 1 + 2 * case["iters"] if k == "newton" else 2
        f, by = one(nn, nc, dim, 1 if dim == 3 else case["nky"], ns, solves, case["dtype"], 3 * nd)
        tot = [tot[0] + f, tot[1] + by]
    return {"bytes": float(tot[1]), "flops": float(tot[0])}


# ------------------------------------------------- float64 restatement (torch)
def _edge_terms(h, s, ky):
    """Edge conductances per axis and the diagonal beyond them (nodal mass and Robin term) of the
    nodal operator for cell conductivities s (batch of shape (nky or 1, *cells))."""
    dim = len(h)
    hw = [torch.as_tensor(w, dtype=_F64, device=DEV) for w in h]
    view = lambda w, a: w.view([1] + [-1 if b == a else 1 for b in range(dim)])  # noqa: E731
    vol = 1.0
    for a in range(dim):
        vol = vol * view(hw[a], a)
    sv = s * vol

    def nodes_from_cells(t, axes):
        for a in axes:
            pad = torch.zeros_like(t.narrow(a + 1, 0, 1))
            t = torch.cat([t, pad], a + 1) + torch.cat([pad, t], a + 1)
        return t

    edges = [nodes_from_cells(sv, [b for b in range(dim) if b != a]) / 2 ** (dim - 1)
             / view(hw[a], a) ** 2 for a in range(dim)]
    diag = 0.0
    if ky is not None:
        k = torch.as_tensor(ky, dtype=_F64, device=DEV).view([-1] + [1] * dim)
        diag = k ** 2 * nodes_from_cells(sv, range(dim)) / 2 ** dim
    x = [torch.as_tensor(v, dtype=_F64, device=DEV) for v in _axes(h)]
    mid = [0.5 * (v[1:] + v[:-1]) for v in x]
    apex = [torch.as_tensor(np.median(np.repeat(v, 1)), dtype=_F64, device=DEV)
            for v in _axes(h)[:-1]] + [torch.zeros((), dtype=_F64, device=DEV)]
    for a in range(dim):
        for side in (0, 1):
            if a == dim - 1 and side == 1:
                continue  # the surface
            # the face centres relative to the top centre of the mesh
            r2, area = 0.0, 1.0
            for b in range(dim):
                p = (x[b][-1 if side else 0] if b == a else view(mid[b], b)) - apex[b]
                r2 = r2 + p ** 2
                if b != a:
                    area = area * view(hw[b], b)
            rdn = (1.0 if side else -1.0) * (x[a][-1 if side else 0] - apex[a])
            r = torch.sqrt(r2)
            if ky is None:
                alpha = rdn / r ** 2
            else:
                kr = k * r
                alpha = (k * torch.special.scaled_modified_bessel_k1(kr)
                         / torch.special.scaled_modified_bessel_k0(kr)) * rdn / r
            face = s.narrow(a + 1, s.shape[a + 1] - 1 if side else 0, 1) * alpha * area
            face = nodes_from_cells(face / 2 ** (dim - 1), [b for b in range(dim) if b != a])
            n = len(h[a])
            zero = torch.zeros_like(face).repeat_interleave(n, dim=a + 1)
            diag = diag + (torch.cat([zero, face], a + 1) if side else torch.cat([face, zero], a + 1))
    return edges, diag


def _apply(edges, diag, u):
    """A u for u of shape (nky, *nodes, sources)."""
    out = diag.unsqueeze(-1) * u
    for a, e in enumerate(edges):
        f = e.unsqueeze(-1) * (u.narrow(a + 1, 1, u.shape[a + 1] - 1)
                               - u.narrow(a + 1, 0, u.shape[a + 1] - 1))
        zero = torch.zeros_like(u.narrow(a + 1, 0, 1))
        out = out - torch.cat([f, zero], a + 1) + torch.cat([zero, f], a + 1)
    return out


class _Slabs:
    """A^{-1} by block elimination over the slabs of the first axis, with one correction."""

    def __init__(self, edges, diag):
        self.edges, self.diag = edges, diag
        nk, nx = diag.shape[0], diag.shape[1]
        inner = diag.shape[2:]
        self.b = b = int(np.prod(inner))
        idx = torch.arange(b, device=DEV).view(inner)
        zero = torch.zeros_like(edges[0].narrow(1, 0, 1))
        main = diag + torch.cat([edges[0], zero], 1) + torch.cat([zero, edges[0]], 1)
        pairs = []
        for a in range(1, len(edges)):
            lo = idx.narrow(a - 1, 0, inner[a - 1] - 1).reshape(-1)
            hi = idx.narrow(a - 1, 1, inner[a - 1] - 1).reshape(-1)
            zero = torch.zeros_like(diag.narrow(a + 1, 0, 1))
            main = main + torch.cat([edges[a], zero], a + 1) + torch.cat([zero, edges[a]], a + 1)
            pairs.append((lo, hi))
        self.e = edges[0].reshape(nk, nx - 1, b)
        self.g = []
        for i in range(nx):
            d = torch.diag_embed(main[:, i].reshape(nk, b))
            for (lo, hi), e in zip(pairs, edges[1:]):
                v = e[:, i].reshape(nk, -1)
                d[:, lo, hi] = -v
                d[:, hi, lo] = -v
            if i:
                d = d - self.e[:, i - 1].unsqueeze(-1) * self.g[-1] * self.e[:, i - 1].unsqueeze(-2)
            self.g.append(torch.linalg.inv(d))

    def _solve(self, rhs):
        shape = rhs.shape
        y = list(rhs.reshape(shape[0], shape[1], self.b, -1).unbind(1))
        for i in range(1, len(y)):
            y[i] = y[i] + self.e[:, i - 1].unsqueeze(-1) * (self.g[i - 1] @ y[i - 1])
        for i in range(len(y) - 1, -1, -1):
            t = y[i] if i + 1 == len(y) else y[i] + self.e[:, i].unsqueeze(-1) * y[i + 1]
            y[i] = self.g[i] @ t
        return torch.stack(y, 1).reshape(shape)

    def solve(self, rhs):
        x = self._solve(rhs)
        return x + self._solve(rhs - _apply(self.edges, self.diag, x))


def exact(case, seed):
    if case["kind"] == "batch":
        return None  # its wavenumbers are fitted by the package
    x = {k: torch.as_tensor(v, device=DEV) for k, v in _inputs(case, seed).items()}
    with torch.no_grad():
        return _exact_solve(case, x) if case["kind"] == "solve" else _exact_survey(case, x)


def _exact_survey(c, x):
    h, a, b, at, m_at, n_at = _geometry(c)
    cells, nodes = [len(w) for w in h], [len(w) + 1 for w in h]
    ky, wq = _wavenumbers(c) if len(h) == 2 else (None, np.ones(1))
    w = torch.as_tensor(wq, device=DEV)
    nk, ns, nd = len(wq), len(a), len(at)

    def grid(v):  # cells numbered with the first axis fastest
        return v.reshape(cells[::-1]).permute(*range(len(cells) - 1, -1, -1)).unsqueeze(0)

    def flat(v):
        return v.squeeze(0).permute(*range(len(cells) - 1, -1, -1)).reshape(-1)

    def spot(nd_idx):  # flat node number (last axis fastest), at the surface
        t = np.zeros(len(nd_idx), np.int64)
        for ax in range(len(nodes)):
            t = t * nodes[ax] + (nodes[ax] - 1 if ax == len(nodes) - 1 else nd_idx[:, ax])
        return torch.as_tensor(t, device=DEV)

    sm, sn = spot(m_at), spot(n_at)
    st = torch.as_tensor(at, device=DEV)
    cr = c["kind"] == "cr"
    mm = x["m"][:x["m"].numel() // 2] if cr else x["m"]
    sig = grid(torch.exp(-mm))
    chg = grid(x["m"][mm.numel():]) if cr else None
    s = sig * (1.0 - 1j * chg) if cr else sig
    edges, diag = _edge_terms(h, s, ky)
    if ky is not None:
        edges = [e.expand(nk, *e.shape[1:]) for e in edges]
    A = _Slabs(edges, diag)
    q = torch.zeros((int(np.prod(nodes)), ns), dtype=s.dtype, device=DEV)
    cols = torch.arange(ns, device=DEV)
    q[spot(a), cols] += 1.0
    if b is not None:
        q[spot(b), cols] -= 1.0
    q = q.reshape(1, *nodes, ns).expand(nk, *nodes, ns)
    U = A.solve(q)

    def project(f):
        t = (w.view(-1, 1, 1) * f.reshape(nk, -1, ns)).sum(0)
        return t[sm, st] - t[sn, st]

    def back(g):  # A^{-1} Pd^T g, the same right-hand side for every wavenumber
        r = torch.zeros((int(np.prod(nodes)), ns), dtype=g.dtype, device=DEV)
        r.index_put_((sm, st), g, accumulate=True)
        r.index_put_((sn, st), -g, accumulate=True)
        return A.solve(r.reshape(1, *nodes, ns).expand(nk, *nodes, ns))

    def sensitivity(g):
        """d/ds of -sum_k w_k y^T A(s) u: the gradient for data cotangent g."""
        y = back(g)
        wk = w.view([-1] + [1] * len(nodes))
        ce = [-wk * ((U.narrow(ax + 1, 1, n - 1) - U.narrow(ax + 1, 0, n - 1))
                     * (y.narrow(ax + 1, 1, n - 1) - y.narrow(ax + 1, 0, n - 1))).sum(-1)
              for ax, n in enumerate(nodes)]
        cd = -wk * (U * y).sum(-1)
        with torch.enable_grad():
            lr = torch.zeros_like(sig).requires_grad_(True)   # d log(rho)
            li = torch.zeros_like(sig).requires_grad_(True)   # d chargeability
            v = sig * torch.exp(-lr)
            v = v * (1.0 - 1j * (chg + li)) if cr else v
            e, dg = _edge_terms(h, v, ky)
            total = sum((p * t).sum() for p, t in zip(e, ce)) + (dg * cd).sum()
            (total.real if cr else total).backward()
        return torch.cat([flat(lr.grad), flat(li.grad)]) if cr else flat(lr.grad)

    V = project(U)
    if c["kind"] == "newton":
        jv, jtu = [], []
        for v in x["v"]:
            e, dg = _edge_terms(h, -sig * grid(v), ky)
            jv.append(project(A.solve(-_apply([t.expand(nk, *t.shape[1:]) for t in e], dg, U))))
        for u in x["u"]:
            jtu.append(sensitivity(u))
        return {"data": V, "Jv": jv, "Jtu": jtu}
    if cr:
        with torch.enable_grad():
            vr, vi = V.real.clone().requires_grad_(True), V.imag.clone().requires_grad_(True)
            d, ip = torch.sqrt(vr ** 2 + vi ** 2), vi / vr
            phi = ((x["w"] * (d - x["dobs"])) ** 2).sum() + ((ip - x["dobs_ip"]) ** 2).sum()
            phi.backward()
        return {"data": d.detach(), "ip": ip.detach(), "phi": phi.detach(),
                "grad": sensitivity(torch.complex(vr.grad, -vi.grad))}
    r = x["w"] * (V - x["dobs"])
    return {"data": V, "phi": (r ** 2).sum(), "grad": sensitivity(2.0 * x["w"] * r)}


def _exact_solve(c, x):
    crow, col, _ = _pattern(c)
    n = len(crow) - 1
    row = torch.as_tensor(np.repeat(np.arange(n), np.diff(crow)), device=DEV)
    col = torch.as_tensor(col.astype(np.int64), device=DEV)
    if c["dtype"] == "float32":  # the values that the solver is given
        x = {k: v.float().double() for k, v in x.items()}
    vals = x["vals"].reshape(c["nbatch"], -1)
    xs, gv, gb = [], [], 0.0
    for i in range(c["nbatch"]):
        A = torch.zeros((n, n), dtype=vals.dtype, device=DEV)
        A[row, col] = vals[i]
        lu, piv = torch.linalg.lu_factor(A)
        b = x["b"]
        sol = torch.linalg.lu_solve(lu, piv, b)
        xs.append(sol + torch.linalg.lu_solve(lu, piv, b - A @ sol))
        if c["grad"]:
            g = x["gx"] if c["nbatch"] == 1 else x["gx"][i]
            adj = torch.linalg.lu_solve(lu, piv, g, adjoint=True)
            adj = adj + torch.linalg.lu_solve(lu, piv, g - A.mH @ adj, adjoint=True)
            gv.append(-(adj[row] * xs[-1].conj()[col]).sum(-1))
            gb = gb + adj
    out = {"x": xs[0] if c["nbatch"] == 1 else torch.stack(xs)}
    if c["grad"]:
        out["grad_vals"] = gv[0] if c["nbatch"] == 1 else torch.stack(gv)
        out["grad_b"] = gb
    return out
