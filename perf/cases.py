"""The calls whose speed matters to a user of the bounding library, with the inputs they meet.

Every case goes through the C entry points of libbqb_gpu.so (include/bqb_gpu.h) the way the reference's host
code and the B&B drivers call them: host arrays in and out where the entry point takes host arrays, device arrays
where it takes those.  Kinds:

  bound      ipm_mc_pk: the basic SDP bound of one problem (the unit of work of every bound)
  batch      bqb_ipm_plan_launch: basic bounds of many subproblems already on the device
  nodes      bqb_bound_nodes_fused: B&B nodes of a graph of at most 128 vertices, a small number of rounds each
  engines    bqb_bound_nodes: B&B nodes above 128 vertices on concurrent engines
  bundle     bundle_method: proximal bundle iterations over a list of triangle cuts
  lambda     lambda_eta: the bundle's inner problem alone
  triangles  getViolated_TriangleInequalities: separation of the most violated triangle inequalities
  rounding   runHeuristic_unpacked: Goemans-Williamson rounding and 1-opt of one X
  kgon       bqb_kgon_sa: pentagonal / heptagonal separation by annealing chains

Node cases stop after one outer round (params.max_outer_iter), as a user who wants many quick bounds sets it: the
bundle's decisions amplify the last digits of X by a factor of ten to a thousand a round, so after some rounds two
correct programs no longer agree to a useful number of digits.  Their incumbent is the best cut a long tabu search finds (a B&B's incumbent is the optimum for
most of its life), so the random streams of the rounding do not change a bound.
"""
import ctypes as C

import numpy as np
import torch

from parallel_biqbin_maxcut_b200 import _lib, instances

IPM_ITERS = 9   # interior-point iterations a basic bound takes at least (7 to 13 over the range)


def listed():
    return [
        # a leaf of a B&B tree: latency of one small bound
        {"name": "bound n=24", "kind": "bound", "graph": "unit", "nv": 24},
        # the root of a dense graph with integer weights
        {"name": "bound n=101", "kind": "bound", "graph": "int", "nv": 101},
        # the root of a 7 x 7 x 7 torus, the largest size of the benchmark (couplings of three decimals)
        {"name": "bound n=343 torus", "kind": "bound", "graph": "torus", "nv": 343, "scale": 1000},
        # first bounds of a benchmark batch: 512 subproblems, 60 to 100 vertices
        {"name": "batch 512 n=60..100", "kind": "batch", "graph": "pm1", "nv": 100, "count": 512, "kmax": 40},
        # a few open nodes early in a tree: fewer nodes than SMs
        {"name": "nodes 16 of n=60", "kind": "nodes", "graph": "unit", "nv": 60, "count": 16, "kmax": 12},
        # the benchmark's batch of nodes
        {"name": "nodes 512 of n=100", "kind": "nodes", "graph": "pm1", "nv": 100, "count": 512, "kmax": 40},
        # nodes of the 150-vertex family, bounded by engines
        {"name": "engines 8 of n=150", "kind": "engines", "graph": "int", "nv": 150, "count": 8, "kmax": 10},
        # a bundle call of a 100-vertex root: one IPM, one lambda_eta and the cut operators an iteration
        {"name": "bundle n=100 m=1500", "kind": "bundle", "graph": "pm1", "nv": 100, "m": 1500, "iters": 5},
        # the inner problem at the size a torus root reaches
        {"name": "lambda m=16000 k=16", "kind": "lambda", "m": 16000, "k": 16},
        # separation at a torus root, the shipped list size
        {"name": "triangles n=343", "kind": "triangles", "graph": "torus", "nv": 343, "T": 5000},
        # rounding at a 100-vertex root
        {"name": "rounding n=100", "kind": "rounding", "graph": "pm1", "nv": 100},
        # heptagonal separation at a 100-vertex root: 4 types, 50 trials each
        {"name": "heptagonal n=100", "kind": "kgon", "graph": "int", "nv": 100, "k": 7, "chains": 200},
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["bound", "bound", "batch", "nodes", "nodes", "engines", "bundle", "lambda", "triangles",
                       "rounding", "kgon"])
    # (the converted QUBOs' last digits are lost in the bounds: they are drawn where none is computed)
    graph = rng.choice(["unit", "pm1", "int"] + (["qubo"] if kind in ("triangles", "rounding", "kgon") else []))
    c = {"kind": kind, "graph": graph}
    if kind == "bound":
        c["nv"] = _log(rng, 16, 343)
        if rng.random() < 0.25:
            c.update(graph="torus", nv=rng.choice([6, 7]) ** 3, scale=rng.randint(10, 999))
    elif kind == "batch":
        c["nv"] = _log(rng, 30, 128)
        c.update(count=_log(rng, 20, 400), kmax=rng.randint(0, c["nv"] // 2 - 1))
    elif kind == "nodes":
        c["nv"] = _log(rng, 30, 110)
        c.update(count=_log(rng, 8, 300), kmax=rng.randint(5, c["nv"] // 2))
    elif kind == "engines":
        c["nv"] = rng.randint(130, 170)
        c.update(count=rng.randint(2, 8), kmax=rng.randint(0, 12))
    elif kind == "bundle":
        c["nv"] = _log(rng, 40, 160)
        c.update(m=_log(rng, 100, min(2500, 20 * c["nv"])), iters=rng.randint(2, 5))
    elif kind == "lambda":
        c.pop("graph")
        c.update(m=_log(rng, 200, 16000), k=rng.randint(2, 24))
    elif kind == "triangles":
        c["nv"] = _log(rng, 30, 343)
        c["T"] = rng.choice([3 * c["nv"], 5000])
    elif kind == "rounding":
        c["nv"] = _log(rng, 30, 200)
    else:
        c["nv"] = _log(rng, 30, 200)
        c.update(k=rng.choice([5, 7]), chains=rng.choice([60, 120, 180]))
    return c


# ---- inputs ------------------------------------------------------------------

def _adjacency(graph, nv, seed, scale=1000):
    if graph == "torus":
        return instances.torus3d(round(nv ** (1 / 3)), seed, scale)
    if graph == "unit":
        return instances.gnp_unit(nv, 0.5, seed)
    if graph == "pm1":
        return instances.gnp_pm1(nv, 0.5, seed)
    if graph == "int":
        return instances.gnp_int(nv, 0.9, 10, seed)
    return instances.qubo_to_maxcut(instances.qubo_dense(nv - 1, 0.1, seed))


def _interior_x(L, seed, share=0.05):
    """A feasible interior X near the solution of the basic bound of L: a low-rank ascent, mixed with the identity."""
    n = L.shape[0]
    W = L - np.diag(np.diag(L))
    rng = np.random.default_rng(seed)
    V = rng.standard_normal((n, int(np.sqrt(2 * n)) + 2))
    V /= np.linalg.norm(V, axis=1, keepdims=True)
    W /= np.abs(W).max()
    shift = 0.5 * np.abs(W).sum(axis=1, keepdims=True) + 1e-3
    for _ in range(150):
        V = shift * V + W @ V
        V /= np.linalg.norm(V, axis=1, keepdims=True)
    X = (1 - share) * (V @ V.T)
    X = 0.5 * (X + X.T)
    np.fill_diagonal(X, 1.0)
    return X


def _tabu_cut(A, seed, starts=512):
    """Best cut value of a tabu search from many starts (the incumbent a B&B holds)."""
    n = A.shape[0]
    g = torch.Generator(device="cuda").manual_seed(seed)
    W = torch.tensor(A, device="cuda")
    x = (torch.rand(starts, n, generator=g, device="cuda") < 0.5).double() * 2 - 1
    gain = x * (x @ W)   # what flipping vertex i adds to the cut
    val = (W.sum() - (x * (x @ W)).sum(1)) / 4
    best = val.clone()
    tabu = torch.zeros(starts, n, device="cuda")
    rows = torch.arange(starts, device="cuda")
    for it in range(12 * n):
        free = torch.where((tabu > it) & (val[:, None] + gain <= best[:, None]), -1e18, gain)
        i = free.argmax(1)
        val = val + gain[rows, i]
        xi = x[rows, i]
        gain[rows, i] = -gain[rows, i]
        gain = gain - 2 * x * W[i] * xi[:, None]
        x[rows, i] = -xi
        tabu[rows, i] = it + 6 + torch.rand(starts, generator=g, device="cuda") * 8
        best = torch.maximum(best, val)
    return float(best.max().round())


def _fixings(nv, count, kmax, seed):
    """Vertices and values fixed at random, the number of them spread evenly over 0..kmax in a fixed shuffled order."""
    ks = np.random.default_rng(7).permutation(np.arange(count) % (kmax + 1))
    rng = np.random.default_rng(seed)
    out = []
    for k in ks:
        xf, sol = np.zeros(nv - 1, np.int32), np.zeros(nv - 1, np.int32)
        at = rng.choice(nv - 1, size=k, replace=False)
        xf[at] = 1
        sol[at] = rng.integers(0, 2, size=k)
        out.append((xf, sol))
    return out


def _subproblem(SPL, xf, sol):
    """The matrix of a node (src/evaluate.c:38-115)."""
    free = np.flatnonzero(xf == 0)
    ones = np.flatnonzero((xf == 1) & (sol == 1))
    S = SPL[np.ix_(free, free)]
    f2 = 2 * SPL[np.ix_(ones, free)].sum(axis=0)
    n = len(free) + 1
    L = np.zeros((n, n))
    L[:-1, :-1] = S + np.diag(f2)
    L[:-1, -1] = L[-1, :-1] = S.sum(axis=1) + f2
    L[-1, -1] = L[-1, :-1].sum()
    return 0.25 * L


class _Plan:
    """The plan of a batch, freed with the object."""

    def __init__(self, lib, Ls, ns):
        self.lib, n = lib, len(ns)
        self.sizes = np.array(ns, np.int32)
        off = np.concatenate([[0], np.cumsum(self.sizes.astype(np.int64) ** 2)])
        self.L = torch.tensor(np.concatenate([L.T.reshape(-1) for L in Ls]), device="cuda")
        self.X = torch.zeros_like(self.L)
        self.out = torch.zeros(n, 4, dtype=torch.float64, device="cuda")
        pl = (C.c_void_p * n)(*[self.L.data_ptr() + 8 * int(o) for o in off[:-1]])
        px = (C.c_void_p * n)(*[self.X.data_ptr() + 8 * int(o) for o in off[:-1]])
        self.stream = torch.cuda.Stream()
        torch.cuda.current_stream().synchronize()
        self.plan = lib.bqb_ipm_plan_create(pl, px, _lib.iptr(self.sizes), n, self.out.data_ptr())

    def __del__(self):
        self.lib.bqb_ipm_plan_destroy(self.plan)


_libc = C.CDLL("libc.so.6")
_NODE = np.dtype([("xfixed", "i4", _lib.NMAX), ("sol", "i4", _lib.NMAX), ("fracsol", "f8", _lib.NMAX),
                  ("level", "i4"), ("pad", "i4"), ("upper_bound", "f8")])


def _params(nv):
    """The benchmark's parameters, one outer round, triangle cuts only."""
    p = dict(_lib.PARAMS_FILE)
    p.update(adjust_TriIneq=0, TriIneq=3 * nv, max_outer_iter=1, extra_iter=0, include_Pent=0, include_Hepta=0)
    return _lib.make_params(**p)


def _triangles(X, m, rng):
    """m violated triangle inequalities of X (the most violated of a random choice), as (type, i, j, k) rows."""
    n = X.shape[0]
    i, j, k = (rng.integers(0, n, 40 * m + 4000) for _ in range(3))
    s = np.sort(np.stack([i, j, k]), axis=0)[::-1]
    s = np.unique(s[:, (s[0] > s[1]) & (s[1] > s[2])], axis=1)
    a, b, c = X[s[0], s[1]], X[s[0], s[2]], X[s[1], s[2]]
    v = np.stack([-a - b - c, -a + b + c, a - b + c, a + b - c]) - 1
    t = v.argmax(axis=0)
    top = np.argsort(-v.max(axis=0), kind="stable")[:m]
    return np.stack([t[top] + 1, s[0, top], s[1, top], s[2, top]], axis=1).astype(np.int32), v.max(axis=0)[top]


_SIGN = np.array([[0, 0, 0, 0], [-1, -1, -1, 0], [-1, 1, 1, 0], [1, -1, 1, 0], [1, 1, -1, 0]])[:, :3]


def _lambda_inputs(c, seed):
    """A bundle of k subgradients over m cuts with the spread, the multipliers and the step a node's bundle has."""
    rng = np.random.default_rng(seed)
    m, k = c["m"], c["k"]
    t = 200.0 / m
    G = 0.25 * rng.standard_normal((m, 1)) + 0.4 * rng.standard_normal((m, k)) + 0.05
    gamma = np.where(rng.random(m) < 0.7, 0.4 * t * rng.exponential(1.0, m), 0.0)
    zeta = -240 + 4 * rng.random(k)
    return G, gamma, zeta, t


def prepare(case, seed):
    lib = _lib.load()
    lib.bqb_init(0)
    kind = case["kind"]
    s = {"lib": lib, "kind": kind}
    if kind == "lambda":
        G, gamma, zeta, t = _lambda_inputs(case, seed)
        m, k = G.shape
        s.update(G=np.ascontiguousarray(G.T), gamma=gamma, zeta=zeta, t0=t, t=C.c_double(),
                 P=_lib.Problem(None, 100, m, 0, 0, k), dgamma=np.zeros(m), eta=np.zeros(m), lam=np.zeros(k))
        return s
    nv = case["nv"]
    A = _adjacency(case["graph"], nv, seed, case.get("scale", 1000))
    if kind == "bound":
        s.update(L=_lib.colmajor(instances.root_matrix(A)), n=nv, X=np.zeros(nv * nv), phi=C.c_double())
    elif kind == "batch":
        SPL = 4 * instances.root_matrix(A)
        Ls = [_subproblem(SPL, xf, sol) for xf, sol in _fixings(nv, case["count"], case["kmax"], seed + 1)]
        s["plan"] = _Plan(lib, Ls, [L.shape[0] for L in Ls])
    elif kind in ("nodes", "engines"):
        nodes = (_lib.BabNode * case["count"])()
        view = np.frombuffer(nodes, _NODE)
        for q, (xf, sol) in enumerate(_fixings(nv, case["count"], case["kmax"], seed + 1)):
            view["xfixed"][q, : nv - 1] = xf
            view["sol"][q, : nv - 1] = sol
            view["level"][q] = xf.sum()
        lb = _tabu_cut(A, seed)
        s.update(A=np.ascontiguousarray(A), nodes=nodes, frac=view["fracsol"][:, : nv - 1], lb=lb, nv=nv, diff=(0.12 if kind == "nodes" else 0.3) * lb,
                 params=_params(nv), bounds=np.zeros(case["count"]))
    elif kind == "bundle":
        rng = np.random.default_rng(seed + 2)
        L = instances.root_matrix(A)
        X = _interior_x(L, seed + 1)
        cuts, viol = _triangles(X, case["m"], rng)
        m = len(cuts)
        g = _lib.GlobalArrays(lib, nv, bundle_cap=case["iters"] + 4, g_rows=m, list_cap=16, cut_cap=m + 16)
        for q, (t, i, j, k) in enumerate(cuts.tolist()):
            g.cuts[q].type, g.cuts[q].i, g.cuts[q].j, g.cuts[q].k = t, i, j, k
        F0 = float((L * X).sum())
        f0 = F0 + 0.02 * abs(F0)
        s.update(glob=g, L=_lib.colmajor(L), X0=_lib.colmajor(X), m=m, F0=F0, f0=f0, iters=case["iters"], n=nv,
                 G0=1.0 - _cut_values(cuts, X), t0=0.5 * 0.1 * f0 / (m * viol.max() ** 2), t=C.c_double())
        s["P"] = _lib.Problem(s["L"].ctypes.data_as(_lib.D), nv, m, 0, 0, 1)
    elif kind == "triangles":
        s.update(X=_lib.colmajor(_interior_x(instances.root_matrix(A), seed + 1)), n=nv, params=_lib.make_params(TriIneq=case["T"]),
                 list=(_lib.TriIneq * case["T"])(), size=C.c_int())
    elif kind == "rounding":
        s.update(X=_lib.colmajor(_interior_x(instances.root_matrix(A), seed + 1)), n=nv, A=A, seed=seed,
                 P0L=_lib.colmajor(4 * instances.root_matrix(A)), PL=_lib.colmajor(instances.root_matrix(A)),
                 xf=np.zeros(nv, np.int32), sol=np.zeros(nv, np.int32), x=np.zeros(nv, np.int32))
    else:
        ch = case["chains"]
        s.update(X=_lib.colmajor(_interior_x(instances.root_matrix(A), seed + 1)), n=nv, k=case["k"], chains=ch, seed=seed,
                 cost=np.zeros(ch), perm=np.zeros(7 * ch, np.int32))
    return s


# ---- the calls ------------------------------------------------------------------

def run(s):
    lib, kind = s["lib"], s["kind"]
    if kind == "bound":
        lib.ipm_mc_pk(_lib.dptr(s["L"]), s["n"], _lib.dptr(s["X"]), C.byref(s["phi"]), 0)
        return {"phi": s["phi"].value, "X": s["X"]}
    if kind == "batch":
        p = s["plan"]
        lib.bqb_ipm_plan_launch(p.plan, p.stream.cuda_stream)
        return {"X": p.X, "phi": p.out[:, 0], "psi": p.out[:, 3], "iterations": p.out[:, 1], "status": p.out[:, 2]}
    if kind in ("nodes", "engines"):
        # the problem, then the batch from the incumbent; diff: what the cuts gained at the root (a node whose basic
        # bound is further than that above the incumbent is given up at once)
        _lib.set_params(lib, s["params"])
        lib.process_adj_matrix(_lib.dptr(s["A"]), s["nv"])
        C.c_double.in_dll(lib, "diff").value = s["diff"]
        lib.bqb_reset_incumbent(s["lb"])
        if kind == "nodes":
            rc = lib.bqb_bound_nodes_fused(s["nodes"], len(s["nodes"]), 1, _lib.dptr(s["bounds"]))
        else:
            rc = lib.bqb_bound_nodes(s["nodes"], len(s["nodes"]), 1, 4, None, _lib.dptr(s["bounds"]))
        return {"bounds": s["bounds"], "fracsol": s["frac"], "rc": rc}
    if kind == "bundle":
        g, P, n, m = s["glob"], s["P"], s["n"], s["m"]
        g.bind()
        g["X"][:] = s["X0"]
        g["X_bundle"][: n * n] = s["X0"]
        g["G"][:m] = s["G0"]
        g["F"][0] = s["F0"]
        g["dual_gamma"][:m] = 0.0
        C.c_double.in_dll(lib, "f").value = s["f0"]
        s["t"].value = s["t0"]
        P.bundle = 1
        lib.bundle_method(C.byref(P), C.byref(s["t"]), s["iters"])
        return {"f": C.c_double.in_dll(lib, "f").value, "t": s["t"].value, "bundle": P.bundle,
                "gamma": g["dual_gamma"][:m], "X": g["X"], "F": g["F"], "G": g["G"]}
    if kind == "lambda":
        s["t"].value = s["t0"]
        d = _lib.dptr
        lib.lambda_eta(C.byref(s["P"]), d(s["zeta"]), d(s["G"]), d(s["gamma"]), d(s["dgamma"]), d(s["lam"]),
                       d(s["eta"]), C.byref(s["t"]))
        return {"dgamma": s["dgamma"], "lambda": s["lam"], "eta": s["eta"], "t": s["t"].value}
    if kind == "triangles":
        _lib.set_params(lib, s["params"])
        top = lib.getViolated_TriangleInequalities(_lib.dptr(s["X"]), s["n"], s["list"], C.byref(s["size"]))
        rows = np.frombuffer(s["list"], np.dtype([("c", "i4", 4), ("value", "f8"), ("y", "f8")]))
        return {"max": top, "size": s["size"].value, "cuts": rows["c"], "values": rows["value"]}
    if kind == "rounding":
        _libc.srand(2020)
        C.c_int.in_dll(lib, "BabPbSize").value = s["n"] - 1
        C.c_void_p.in_dll(lib, "X").value = s["X"].ctypes.data
        v = lib.runHeuristic_unpacked(_lib.dptr(s["P0L"]), s["n"], _lib.dptr(s["PL"]), s["n"], _lib.iptr(s["xf"]),
                                      _lib.iptr(s["sol"]), _lib.iptr(s["x"]))
        return {"value": v, "x": s["x"][: s["n"] - 1]}
    rc = lib.bqb_kgon_sa(_lib.dptr(s["X"]), s["n"], s["k"], 3 if s["k"] == 5 else 4, s["chains"], s["seed"],
                         _lib.dptr(s["cost"]), _lib.iptr(s["perm"]))
    return {"rc": rc, "cost": s["cost"], "perm": s["perm"]}


# ---- what a pass cannot do without ----------------------------------------------------

def _ipm_flops(n, iters=IPM_ITERS):
    """Two products 4 n^3, inv(Z) n^3, the Cholesky factor of Zi .* X n^3 / 3, two line-search factors 2 n^3 / 3."""
    return 6.0 * iters * float(n) ** 3


def work(case):
    kind = case["kind"]
    if kind == "lambda":
        m, k = case["m"], case["k"]
        # Q = t G'G, then about 8 rounds of G'eta and G lambda
        return {"bytes": 8 * (m * k + 3 * m), "flops": m * k * (k + 1) + 8 * 4 * m * k + 8 * 12 * 2 * k ** 3 / 3}
    n = case["nv"]
    if kind == "bound":
        return {"bytes": 16 * n * n, "flops": _ipm_flops(n)}
    if kind == "batch":
        na = n - case["kmax"] / 2
        return {"bytes": 16 * na * na * case["count"], "flops": _ipm_flops(na) * case["count"]}
    if kind in ("nodes", "engines"):
        # a basic bound and one rounding (a factor, n hyperplanes) for every node
        na = n - case["kmax"] / 2
        return {"bytes": case["count"] * 16 * n, "flops": case["count"] * (_ipm_flops(na) + 2.4 * na ** 3)}
    if kind == "bundle":
        m, it = case["m"], case["iters"]
        return {"bytes": 8 * (2 * n * n + m * (it + 4)) + 16 * m, "flops": it * (_ipm_flops(n) + 40 * m)}
    if kind == "triangles":
        c = n * (n - 1) * (n - 2) / 6
        return {"bytes": 8 * n * n + 24 * case["T"], "flops": 4 * 4 * c}
    if kind == "rounding":
        # two factors, two rounds of n hyperplanes: projection, 1-opt products, evaluation
        return {"bytes": 24 * n * n, "flops": 2 * (n ** 3 / 3 + 5.0 * n ** 3)}
    return {"bytes": 8 * n * n, "flops": case["chains"] * 3000.0 * n * case["k"] / 10}


# ---- the same results in 64 bits, without the library ------------------------------------

def _pd(M):
    try:
        np.linalg.cholesky(M)
        return True
    except np.linalg.LinAlgError:
        return False


def _ipm(L):
    """The predictor-corrector method of the basic bound: (X, phi, psi, iterations)."""
    n = L.shape[0]
    y = np.abs(L).sum(axis=0) + 1.1
    X, Z = np.eye(n), np.diag(y) - L
    phi, psi, mu, it = y.sum(), np.trace(L), np.trace(Z) / (2 * n), 0
    while abs(phi - psi) > 1e-2:
        it += 1
        Zi = np.linalg.inv(Z)
        Zi = 0.5 * (Zi + Zi.T)
        M = Zi * X
        d1 = np.linalg.solve(M, -np.ones(n))
        D1 = Zi @ (-d1[:, None] * X) - X
        D1 = 0.5 * (D1 + D1.T)
        d2 = np.linalg.solve(M, mu * np.diag(Zi) - (Zi * D1) @ d1)
        D = D1 + Zi @ (-d2[:, None] * X - d1[:, None] * D1) + mu * Zi
        D = 0.5 * (D + D.T)
        dy, ap, ad = d1 + d2, 1.0, 1.0
        while not _pd(X + ap * D):
            ap *= 0.8
        while not _pd(Z + ad * np.diag(dy)):
            ad *= 0.8
        ap, ad = (0.95 * ap if ap < 1 else ap), (0.95 * ad if ad < 1 else ad)
        X, y, Z = X + ap * D, y + ad * dy, Z + ad * np.diag(dy)
        mu = (Z * X).sum() / (2 * n)
        mu *= (0.5 if ap + ad > 1.6 else 1.0) * (0.2 if ap + ad > 1.9 else 1.0)
        phi, psi = y.sum(), (L * X).sum()
    return X, phi, psi, it


def _cut_values(cuts, X):
    """B(X): the left-hand side s_ij X_ij + s_ik X_ik + s_jk X_jk of every triangle cut (<= 1)."""
    t, i, j, k = cuts.T
    s = _SIGN[t]
    return s[:, 0] * X[i, j] + s[:, 1] * X[i, k] + s[:, 2] * X[j, k]


def _qp(Q, c):
    """The simplex-constrained QP of the bundle."""
    k = len(c)
    lam = np.full(k, 1.0 / k)
    w = Q @ lam + c
    y = 0.0 if w.min() > 1 else w.min() - 1.0
    z, Ql = w - y, Q @ lam
    mu, res = 0.5 * (z @ lam) / k, 1.0 - lam.sum()
    cnt = 0
    while abs(lam @ c + lam @ Ql - y) > 1e-5 and cnt <= 30:
        cnt += 1
        A = Q + np.diag(z / lam)
        u, v = np.linalg.solve(A, np.stack([np.ones(k), c - y + Ql]).T).T
        dy = (res + v.sum()) / u.sum()
        dl = u * dy - v
        dz = (mu - lam * z - z * dl) / lam
        ap, ad = (-dl / lam).max(), (-dz / z).max()
        ap, ad = (min(0.99 / a, 1.0) if a > 0 else 1.0 for a in (ap, ad))
        y, lam, z = y + ad * dy, lam + ap * dl, z + ad * dz
        res, Ql, mu = 1 - lam.sum(), Q @ lam, 0.4 * (lam @ z) / k * (0.2 if ap + ad > 1.8 else 1.0)
    return lam


def _lambda_eta(zeta, G, gamma, t):
    eta, Q, last, cnt = np.zeros(G.shape[0]), t * (G.T @ G), 0.0, 0
    while True:
        cnt += 1
        lam = _qp(Q, zeta - t * (G.T @ eta))
        w = G @ lam
        eta = np.maximum(w - gamma / t, 0.0)
        d = t * (eta - w)
        now = np.linalg.norm(d)
        if cnt >= 50:
            return d, lam, eta, t * 0.95
        if abs(now - last) / (1 + now) < 1e-5:
            return d, lam, eta, t
        last = now


def exact(case, seed):
    kind = case["kind"]
    if kind == "lambda":
        d, lam, eta, t = _lambda_eta(*(lambda G, gamma, zeta, t: (zeta, G, gamma, t))(*_lambda_inputs(case, seed)))
        return {"dgamma": d, "lambda": lam, "eta": eta, "t": t}
    if kind not in ("bound", "batch"):
        return None   # whole numbers, or a chain of discrete decisions
    nv = case["nv"]
    A = _adjacency(case["graph"], nv, seed, case.get("scale", 1000))
    if kind == "bound":
        X, phi, _, _ = _ipm(instances.root_matrix(A))
        return {"phi": float(phi), "X": X.T.reshape(-1)}
    SPL = 4 * instances.root_matrix(A)
    res = [_ipm(_subproblem(SPL, xf, sol)) for xf, sol in _fixings(nv, case["count"], case["kmax"], seed + 1)]
    return {"X": np.concatenate([r[0].T.reshape(-1) for r in res]), "phi": np.array([r[1] for r in res]),
            "psi": np.array([r[2] for r in res]), "iterations": np.array([float(r[3]) for r in res]),
            "status": np.zeros(len(res))}
