"""Performance cases: what a user of the framework has it do, by size and form.

Five kinds of call, each through the package's public entry points:

* ``stages``: the operator stages (metrics, base-flow derivatives, assembly,
  boundary rows) of a new (alpha, Re) on a grid whose context is kept, and one
  product with each assembled operator;
* ``point``: one stability point, stages and shift-and-invert eigen solve, in
  the mixed form (precision 1) or the plain FP64 form (precision 0);
* ``sweep``: a batched alpha sweep over grid classes with warm starts;
* ``pencil``: an explicit dense pencil A x = lambda B x;
* ``mlp``: the learned proposal's loss and parameter gradients on a batch.

Grids, physics and solver settings come from the repository's benchmark, its
tests and its sweep configurations; the seed moves each case inside the range
it stands for (wavenumber, Reynolds number, wall phase, vectors, pencils,
batches).
"""
from __future__ import annotations

import math

import numpy as np

from tailor_gb300 import api, learned
from tailor_gb300.case import Physics, make_case


def listed():
    return [
        # one (alpha, Re) step of a parameter study on the smallest sweep grid:
        # launches and host round trips, hardly any data
        {"name": "stages_60x32", "kind": "stages", "ny": 60, "nz": 32, "mach": 0.5},
        # the same on the largest grid, where writing the operators counts
        {"name": "stages_300x192", "kind": "stages", "ny": 300, "nz": 192, "mach": 0.7},
        # a point of a small-grid sweep: latency of every dependent step
        {"name": "point_60x32_mixed", "kind": "point", "ny": 60, "nz": 32, "nev": 8, "ncv": 0,
         "alpha": 2.0, "reynolds": 1000.0, "mach": 0.5, "omega_re": 0.0, "omega_im": 0.0,
         "amplitude": 0.05, "precision": 1},
        # a ragged grid (no shipped rule, no multiple of a tile), few pairs,
        # target off the origin
        {"name": "point_83x47_mixed", "kind": "point", "ny": 83, "nz": 47, "nev": 5, "ncv": 0,
         "alpha": 1.3, "reynolds": 800.0, "mach": 0.3, "omega_re": 0.1, "omega_im": 0.0,
         "amplitude": 0.03, "precision": 1},
        # the ordinary single-case grid
        {"name": "point_100x50_mixed", "kind": "point", "ny": 100, "nz": 50, "nev": 8, "ncv": 0,
         "alpha": 2.43, "reynolds": 1000.0, "mach": 0.5, "omega_re": 0.0, "omega_im": 0.0,
         "amplitude": 0.05, "precision": 1},
        # a resolved case with more wanted pairs around a complex target
        {"name": "point_200x128_mixed", "kind": "point", "ny": 200, "nz": 128, "nev": 16,
         "ncv": 64, "alpha": 1.8, "reynolds": 1000.0, "mach": 0.5, "omega_re": 0.3,
         "omega_im": 0.01, "amplitude": 0.08, "precision": 1},
        # a point of the neutral-curve sweep on its grid, the largest case
        {"name": "point_300x192_mixed", "kind": "point", "ny": 300, "nz": 192, "nev": 4,
         "ncv": 64, "alpha": 2.8, "reynolds": 1200.0, "mach": 0.7, "omega_re": 0.0,
         "omega_im": 0.0, "amplitude": 0.05, "precision": 1},
        # the drop-in FP64 form on the smallest sweep grid
        {"name": "point_60x32_fp64", "kind": "point", "ny": 60, "nz": 32, "nev": 8, "ncv": 0,
         "alpha": 2.0, "reynolds": 1000.0, "mach": 0.5, "omega_re": 0.0, "omega_im": 0.0,
         "amplitude": 0.05, "precision": 0},
        # the FP64 form where the factorisation's arithmetic counts
        {"name": "point_150x64_fp64", "kind": "point", "ny": 150, "nz": 64, "nev": 8, "ncv": 0,
         "alpha": 1.6, "reynolds": 1000.0, "mach": 0.5, "omega_re": 0.0, "omega_im": 0.0,
         "amplitude": 0.05, "precision": 0},
        # a batch of instances over two grid classes, contexts made by the call
        {"name": "sweep_12_points", "kind": "sweep", "points": 12, "workers": 4, "nev": 8,
         "ncv": 32},
        # an independently known pencil, no multiple of the block size
        {"name": "pencil_303_fp64", "kind": "pencil", "n": 303, "nev": 6, "precision": 0},
        # one full-batch gradient of the proposal network on a training set
        {"name": "mlp_gradients_2048", "kind": "mlp", "rows": 2048},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["stages", "point", "point", "point", "fp64", "fp64", "sweep", "pencil",
                       "mlp"])
    if kind == "stages":
        return {"kind": "stages", "ny": round(_log(rng, 24, 300)), "nz": round(_log(rng, 16, 192)),
                "mach": round(rng.uniform(0.2, 0.8), 3)}
    if kind in ("point", "fp64"):
        top = (220, 130) if kind == "point" else (130, 60)
        return {"kind": "point", "ny": round(_log(rng, 30, top[0])),
                "nz": round(_log(rng, 18, top[1])), "nev": rng.randint(3, 12), "ncv": 0,
                "alpha": round(rng.uniform(0.8, 3.5), 3),
                "reynolds": round(_log(rng, 600.0, 2400.0), 1),
                "mach": round(rng.uniform(0.3, 0.7), 3), "omega_re": round(rng.uniform(0, 0.3), 3),
                "omega_im": 0.0, "amplitude": round(rng.uniform(0.02, 0.08), 3),
                "precision": 1 if kind == "point" else 0}
    if kind == "sweep":
        return {"kind": "sweep", "points": rng.randint(4, 12), "workers": rng.randint(1, 6),
                "nev": rng.randint(4, 10), "ncv": 32}
    if kind == "pencil":
        return {"kind": "pencil", "n": round(_log(rng, 12, 600)), "nev": rng.randint(1, 5),
                "precision": rng.choice([0, 1])}
    return {"kind": "mlp", "rows": round(_log(rng, 24, 2048))}


def _rng(case, seed):
    # the sizes take part, so that equal seeds of two cases are unrelated
    sizes = [int(v) for v in case.values() if isinstance(v, int)]
    return np.random.default_rng([int(seed)] + sizes)


def _physics(case, rng):
    j = rng.uniform(-1.0, 1.0, 2)
    return Physics(alpha=case.get("alpha", 1.7) * (1.0 + 0.04 * j[0]),
                   reynolds=case.get("reynolds", 1000.0) * (1.0 + 0.05 * j[1]),
                   mach=case["mach"],
                   omega=complex(case.get("omega_re", 0.0), case.get("omega_im", 0.0)),
                   nev=case.get("nev", 8), tol=1e-10)


def _pencil(case, seed):
    """A random non-normal A, and B block diagonal in 5 x 5 blocks."""
    n = case["n"]
    r = _rng(case, seed)
    c = lambda *s: r.standard_normal(s) + 1j * r.standard_normal(s)  # noqa: E731
    a = c(n, n) / math.sqrt(2 * n)
    b = np.zeros((n, n), complex)
    for i in range(0, n, 5):
        k = min(5, n - i)
        b[i:i + k, i:i + k] = np.eye(k) + 0.1 * c(k, k)
    # a search centre inside the spectrum's disk
    return a, b, complex(0.3, -0.2) + 0.1 * complex(*r.standard_normal(2))


def _batch(case, seed):
    """Training rows: (alpha, log10 Re, Mach), smooth targets with noise;
    parameters scaled as the network's own initialisation."""
    r = _rng(case, seed)
    n = case["rows"]
    x = np.stack([r.uniform(0.5, 4.0, n), r.uniform(2.7, 3.5, n), r.uniform(0.2, 0.8, n)],
                 1).astype(np.float32)
    y = (np.sin(x @ r.standard_normal((3, 80))) + 0.05 * r.standard_normal((n, 80))
         ).astype(np.float32)
    dims = [3, 256, 256, 256, 256, 80]
    params = np.concatenate([
        np.concatenate([(r.standard_normal(o * i) / math.sqrt(i)), 0.1 * r.standard_normal(o)])
        for i, o in zip(dims, dims[1:])]).astype(np.float32)
    return x, y, params, dims


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("stages", "point"):
        r = _rng(case, seed)
        ph = _physics(case, r)
        grid = make_case(case["ny"], case["nz"], amplitude=case.get("amplitude", 0.05),
                         seed=int(r.integers(1, 1 << 30)), physics=ph)
        state = {"case": case, "problem": api.Problem(grid), "physics": ph}
        if kind == "stages":
            n = 5 * grid.nodes
            state["x"] = r.standard_normal(n) + 1j * r.standard_normal(n)
        return state
    if kind == "sweep":
        r = _rng(case, seed)
        grids = [make_case(60, 32, seed=int(r.integers(1, 1 << 30)),
                           physics=Physics(nev=case["nev"], tol=1e-10)),
                 make_case(100, 50, seed=int(r.integers(1, 1 << 30)),
                           physics=Physics(nev=case["nev"], tol=1e-10))]
        alphas = np.sort(r.uniform(0.8, 3.5, case["points"]))
        # two thirds of the points on the smaller grid
        points = [(1 if i >= (2 * case["points"]) // 3 else 0, complex(a))
                  for i, a in enumerate(alphas)]
        return {"case": case, "grids": grids, "points": points}
    if kind == "pencil":
        a, b, centre = _pencil(case, seed)
        return {"case": case, "A": a, "B": b, "centre": centre}
    x, y, params, _ = _batch(case, seed)
    net = learned.MLP()
    net.set_params(params)
    return {"case": case, "net": net, "x": x, "y": y}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("stages", "point"):
        p = state["problem"]
        p.set_physics(state["physics"])
        api.run_pipeline(p)
        if kind == "stages":
            x = state["x"]
            return {"Ax": p.spmv(api.TLR_MAT_A, x), "Bx": p.spmv(api.TLR_MAT_B, x)}
        sol = api.EigenSolver(p).solve(nev=case["nev"], ncv=case["ncv"],
                                       precision=case["precision"])
        return {"lam": sol.lam}
    if kind == "sweep":
        res = api.sweep(state["grids"], state["points"], nev=case["nev"], ncv=case["ncv"],
                        precision=1, workers=case["workers"], warm_start=True)
        return {"lam": res.lam, "status": res.status}
    if kind == "pencil":
        z = state["centre"]  # lambda_s = Im(omega) - i Re(omega)
        sol = api.solve_pencil(state["A"], state["B"], omega=complex(-z.imag, z.real),
                               nev=case["nev"], precision=case["precision"], modes=False)
        return {"lam": sol.lam}
    loss, grads = state["net"].gradients(state["x"], state["y"])
    return {"loss": np.float32(loss), "grads": grads}


def _operator_bytes(nodes):
    # per node: 3 + 5 complex fields in, and per operator pair 77 blocks of A
    # and one of B, 400 bytes each, written once
    return nodes * (8 * 16 + 78 * 400)


def _point_work(ny, nz, nev, ncv, precision):
    rules = make_case(ny, nz)
    s = api.symbolic_analysis(rules.xi, rules.eta)
    entry = 8 if precision else 16
    applications = ncv or max(2 * nev, nev + 15)
    return {"bytes": _operator_bytes(ny * nz) + s["factor_elems"] * entry * (1 + applications),
            "flops": s["flops"] + 8.0 * s["factor_elems"] * applications}


def work(case):
    kind = case["kind"]
    if kind == "stages":
        nodes = case["ny"] * case["nz"]
        # the operators written and read once (one product), two vectors in
        # and out; the node coefficients' arithmetic is about 30 kflop
        return {"bytes": 2 * _operator_bytes(nodes) + 4 * 80 * nodes,
                "flops": nodes * (30e3 + 78 * 200)}
    if kind == "point":
        return _point_work(case["ny"], case["nz"], case["nev"], case["ncv"], case["precision"])
    if kind == "sweep":
        small = (2 * case["points"]) // 3
        w = [_point_work(60, 32, case["nev"], case["ncv"], 1),
             _point_work(100, 50, case["nev"], case["ncv"], 1)]
        return {k: small * w[0][k] + (case["points"] - small) * w[1][k] for k in w[0]}
    if kind == "pencil":
        n = case["n"]
        return {"bytes": 32.0 * n * n, "flops": 8.0 / 3.0 * n ** 3}
    weights = 3 * 256 + 3 * 256 * 256 + 256 * 80
    return {"bytes": 4.0 * (case["rows"] * 83 + 2 * (weights + 4 * 256 + 80)),
            "flops": 6.0 * case["rows"] * weights}


def exact(case, seed):
    """Pencils: numpy's dense eigenvalues nearest the centre.  Gradients: the
    network in 64 bits.  The grid kinds have none: their eigenvalues take a
    sparse FP64 factorisation of minutes on the host."""
    if case["kind"] == "pencil":
        a, b, z = _pencil(case, seed)
        lam = np.linalg.eigvals(np.linalg.solve(b, a))
        return {"lam": lam[np.argsort(np.abs(lam - z))][:case["nev"]]}
    if case["kind"] == "mlp":
        x, y, params, dims = _batch(case, seed)
        x, y, params = x.astype(np.float64), y.astype(np.float64), params.astype(np.float64)
        layers, at = [], 0
        for i, o in zip(dims, dims[1:]):
            layers.append((params[at:at + o * i].reshape(o, i), params[at + o * i:at + o * i + o]))
            at += o * i + o
        acts, pre = [x], []
        for k, (w, b) in enumerate(layers):
            z = acts[-1] @ w.T + b
            pre.append(z)
            acts.append(z / (1.0 + np.exp(-z)) if k + 1 < len(layers) else z)
        d = acts[-1] - y
        g = 2.0 * d / d.size
        grads = []
        for k in reversed(range(len(layers))):
            if k + 1 < len(layers):
                s = 1.0 / (1.0 + np.exp(-pre[k]))
                g = g * (s * (1.0 + pre[k] * (1.0 - s)))
            grads.insert(0, np.concatenate([(g.T @ acts[k]).ravel(), g.sum(0)]))
            g = g @ layers[k][0]
        return {"loss": np.float64((d * d).mean()), "grads": np.concatenate(grads)}
    return None
