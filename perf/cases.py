"""The work that programs built on this solver have it do, as measurable cases.

Every case goes through the public Python classes (``RGF``, ``RGFBatch``), on
seeded block-tridiagonal-arrowhead matrices of the family that
``rgf_gb300.gen`` describes, built on the GPU here so that large ones are
quick to make:

* ``evaluate``: a handle is kept and one evaluation is factorize + logDet +
  RGFdiag (what each step of a hyper-parameter search or a model fit needs);
* ``solve``: right-hand sides against a factor that stays resident;
* ``batch``: many uneven instances evaluated together;
* ``oneshot``: a new matrix from host arrays to its results, the handle
  created and closed inside the pass (the flow of the reference's main program).
"""
import math

import numpy as np
import torch

import rgf_gb300
from rgf_gb300.flops import algorithmic_flops

# sizes of the batched workload's classes
BATCH_NS = (42, 128, 256, 512)
BATCH_ND = (0, 2, 6)
# a drawn case costs no more than the largest listed ones (algorithmic flops)
FP64_FLOPS = 4.2e11
SPLIT_FLOPS = 6.5e12


def listed():
    return [
        # the smallest instance: a first try, a unit test, a toy model; every
        # result of the class is asked for (all launches and latency)
        {"name": "tiny_fp64", "kind": "evaluate", "precision": "fp64", "ns": 3, "nt": 3, "nd": 2,
         "spde": False, "want": "all", "nrhs": 1},
        # a small space-time model, with the covariances of neighbouring time
        # steps (the selected inverse's blocks) read back
        {"name": "small_fp64_cov", "kind": "evaluate", "precision": "fp64", "ns": 42, "nt": 30,
         "nd": 6, "spde": False, "want": "cov", "nrhs": 0},
        # many short time steps: long chains of small blocks, split precision
        {"name": "small_split", "kind": "evaluate", "precision": "split", "ns": 128, "nt": 60,
         "nd": 2, "spde": False, "want": "diag", "nrhs": 0},
        # an odd block size with an odd arrowhead in FP64
        {"name": "odd_fp64", "kind": "evaluate", "precision": "fp64", "ns": 333, "nt": 17, "nd": 5,
         "spde": False, "want": "diag", "nrhs": 0},
        # a mid-size model in split precision, ragged against every tile width
        {"name": "mid_split", "kind": "evaluate", "precision": "split", "ns": 515, "nt": 40,
         "nd": 3, "spde": False, "want": "diag", "nrhs": 0},
        # the SPDE-like operator on a 40 x 25 grid over 50 time steps, in both precisions
        {"name": "spde1000_fp64", "kind": "evaluate", "precision": "fp64", "ns": 1000, "nt": 50,
         "nd": 4, "spde": True, "want": "diag", "nrhs": 0},
        {"name": "spde1000_split", "kind": "evaluate", "precision": "split", "ns": 1000, "nt": 50,
         "nd": 4, "spde": True, "want": "diag", "nrhs": 0},
        # the benchmark's instance, the largest
        {"name": "large_split", "kind": "evaluate", "precision": "split", "ns": 2000, "nt": 100,
         "nd": 6, "spde": False, "want": "diag", "nrhs": 0},
        # eight right-hand sides on a resident split factor, refined in FP64
        {"name": "solve8_split", "kind": "solve", "precision": "split", "ns": 1000, "nt": 50,
         "nd": 4, "spde": True, "want": "x", "nrhs": 8},
        # one right-hand side on a resident FP64 factor (a conditional mean)
        {"name": "solve1_fp64", "kind": "solve", "precision": "fp64", "ns": 256, "nt": 60, "nd": 2,
         "spde": False, "want": "x", "nrhs": 1},
        # uneven instances of a parameter search, evaluated as one batch
        {"name": "batch32_split", "kind": "batch", "precision": "split", "count": 32,
         "nt_max": 60, "shape_seed": 7},
        # a new matrix per pass, from host arrays to results
        {"name": "oneshot_split", "kind": "oneshot", "precision": "split", "ns": 256, "nt": 20,
         "nd": 2, "spde": False, "want": "diag", "nrhs": 0},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evaluate"] * 5 + ["solve"] * 2 + ["batch", "oneshot"])
    precision = rng.choice(["fp64", "split"])
    while kind == "batch":
        case = {"kind": "batch", "precision": precision, "count": _log_int(rng, 2, 32),
                "nt_max": _log_int(rng, 4, 60), "shape_seed": rng.randrange(1 << 20)}
        if work(case)["flops"] <= FP64_FLOPS:
            return case
    while True:
        ns = _log_int(rng, 3, 600 if kind == "oneshot" else 2000)
        nt = _log_int(rng, 3, 100)
        nd = rng.randint(0, 6)
        limit = FP64_FLOPS if precision == "fp64" else SPLIT_FLOPS
        if kind == "oneshot":
            limit = 3e10
        if algorithmic_flops(ns, nt, nd)["total"] <= limit:
            break
    case = {"kind": kind, "precision": precision, "ns": ns, "nt": nt, "nd": nd, "spde": False,
            "want": "x" if kind == "solve" else "diag", "nrhs": 0}
    if kind == "solve":
        case["nrhs"] = _log_int(rng, 1, 16)
    elif kind == "evaluate" and ns * ns * nt < 4e6 and rng.random() < 0.5:
        case["want"], case["nrhs"] = rng.choice([("cov", 0), ("all", 1), ("all", 3)])
    return case


# ---- the matrices ------------------------------------------------------------

def _grid(ns):
    """The most nearly square gx * gy = ns (1000: 25 x 40)."""
    g = int(math.isqrt(ns))
    while ns % g:
        g -= 1
    return g, ns // g


def _blocks(ns, nt, nd, spde, seed):
    """D (nt, ns, ns; symmetric), B (nt-1, ns, ns), C (nt, nd, ns), corner (nd, nd)
    as float64 GPU tensors:
    D_i = A_i A_i^T / ns + (ns + 2) I (+ I + 5-point Laplacian), B_i ~ N(0, 0.1 / ns),
    C_i ~ N(0, 0.1), corner = R R^T / nd + (nt + 2) I."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape, dtype=torch.float64):
        return torch.randn(*shape, generator=g, device="cuda", dtype=dtype)

    D = torch.empty(nt, ns, ns, dtype=torch.float64, device="cuda")
    for i in range(nt):
        A = normal(ns, ns, dtype=torch.float32)
        D[i] = A @ A.T
    D /= ns
    D += torch.tril(D, -1).transpose(1, 2) - torch.triu(D, 1)  # exactly symmetric
    D.diagonal(dim1=1, dim2=2).add_(ns + 2.0)
    if spde:
        gx, gy = _grid(ns)
        lap = 5.0 * torch.eye(ns, dtype=torch.float64, device="cuda")
        idx = torch.arange(ns, device="cuda").reshape(gy, gx)
        for p, q in ((idx[:, :-1], idx[:, 1:]), (idx[:-1, :], idx[1:, :])):
            lap[p.reshape(-1), q.reshape(-1)] = -1.0
            lap[q.reshape(-1), p.reshape(-1)] = -1.0
        D += lap
    B = normal(nt - 1, ns, ns) * math.sqrt(0.1 / ns)
    C = normal(nt, nd, ns) * math.sqrt(0.1)
    R = normal(nd, nd)
    corner = R @ R.T / max(nd, 1) + (nt + 2.0) * torch.eye(nd, dtype=torch.float64, device="cuda")
    corner = torch.tril(corner) + torch.tril(corner, -1).T
    return D, B, C, corner


def _csc(ns, nt, nd, blocks):
    """The lower triangle as host CSC arrays (ia, ja: uint64, a: float64)."""
    D, B, C, corner = blocks
    n = ns * nt + nd
    nnz = nt * ns * (ns + 1) // 2 + (nt - 1) * ns * ns + nt * ns * nd + nd * (nd + 1) // 2
    a = torch.empty(nnz, dtype=torch.float64, device="cuda")
    ja = torch.empty(nnz, dtype=torch.int64, device="cuda")
    counts = torch.empty(n, dtype=torch.int64, device="cuda")
    col = torch.arange(ns, device="cuda")
    dense = nt * ns + torch.arange(nd, device="cuda")
    pos = 0
    for i in range(nt):
        parts, rows = [D[i]], [i * ns + col]  # D is symmetric: row c holds column c
        if i < nt - 1:
            parts.append(B[i].T)
            rows.append((i + 1) * ns + col)
        parts.append(C[i].T)
        rows.append(dense)
        panel, row = torch.cat(parts, 1), torch.cat(rows)
        keep = row[None, :] >= (i * ns + col)[:, None]
        k = ns * (ns + 1) // 2 + (row.numel() - ns) * ns
        a[pos:pos + k] = panel[keep]
        ja[pos:pos + k] = row.expand(ns, -1)[keep]
        counts[i * ns:(i + 1) * ns] = row.numel() - col
        pos += k
    if nd:
        keep = torch.ones(nd, nd, dtype=torch.bool, device="cuda").triu()
        a[pos:] = corner[keep]
        ja[pos:] = dense.expand(nd, -1)[keep]
        counts[nt * ns:] = nd - torch.arange(nd, device="cuda")
    ia = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(counts, 0, out=ia[1:])
    return (ia.cpu().numpy().view(np.uint64), ja.cpu().numpy().view(np.uint64), a.cpu().numpy())


def _rhs(n, nrhs, seed):
    rng = np.random.default_rng(seed + 1000003)
    return np.asfortranarray(rng.standard_normal((n, nrhs)))


def _batch_shapes(case):
    rng = np.random.default_rng(case["shape_seed"])
    return [(int(rng.choice(BATCH_NS)), int(rng.integers(3, case["nt_max"] + 1)),
             int(rng.choice(BATCH_ND))) for _ in range(case["count"])]


def _matrix(case, seed):
    sizes = case["ns"], case["nt"], case["nd"]
    return _csc(*sizes, _blocks(*sizes, case["spde"], seed))


# ---- the passes --------------------------------------------------------------

def prepare(case, seed):
    if case["kind"] == "batch":
        inst = []
        for i, (ns, nt, nd) in enumerate(_batch_shapes(case)):
            inst.append((*_csc(ns, nt, nd, _blocks(ns, nt, nd, False, seed * 1009 + i)), ns, nt, nd))
        torch.cuda.empty_cache()
        return {"case": case, "solver": rgf_gb300.RGFBatch(inst, precision=case["precision"])}
    csc = _matrix(case, seed)
    torch.cuda.empty_cache()  # the solver allocates from the driver
    sizes = case["ns"], case["nt"], case["nd"]
    state = {"case": case}
    if case["kind"] == "oneshot":
        state["csc"] = csc
        return state
    state["solver"] = rgf_gb300.RGF(*csc, *sizes, precision=case["precision"])
    if case["nrhs"]:
        state["b"] = _rhs(case["ns"] * case["nt"] + case["nd"], case["nrhs"], seed)
    if case["kind"] == "solve":
        state["solver"].factorize()
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        logdet, diags = state["solver"].run()
        return {"logdet": logdet, "diag": diags}
    if case["kind"] == "oneshot":
        with rgf_gb300.RGF(*state["csc"], case["ns"], case["nt"], case["nd"],
                           precision=case["precision"]) as s:
            s.factorize()
            return {"logdet": np.array([s.logDet()]), "diag": s.RGFdiag()}
    s = state["solver"]
    if case["kind"] == "solve":
        return {"x": s.solve(np.empty_like(state["b"]), state["b"], case["nrhs"])}
    s.factorize()
    out = {"logdet": np.array([s.logDet()])}
    if case["want"] == "all":
        out["x"] = s.solve(np.empty_like(state["b"]), state["b"], case["nrhs"])
        out["factor"] = s.export_factor()
    out["diag"] = s.RGFdiag()
    if case["want"] == "cov":
        out["cov"] = s.export_selinv()
    return out


def _sizes(case):
    if case["kind"] == "batch":
        return _batch_shapes(case)
    return [(case["ns"], case["nt"], case["nd"])]


def work(case):
    """One pass's inputs read once, outputs written once; LAPACK-convention flops."""
    nbytes = flops = 0.0
    for ns, nt, nd in _sizes(case):
        n = ns * nt + nd
        nnz = nt * ns * (ns + 1) // 2 + (nt - 1) * ns * ns + nt * ns * nd + nd * (nd + 1) // 2
        nrhs = case.get("nrhs", 0)
        if case["kind"] != "solve":
            nbytes += 16.0 * nnz + 8.0 * (n + 1) + 8.0 * (n + 1)  # CSC; diag and logDet
            flops += algorithmic_flops(ns, nt, nd)["total"]
            if case.get("want") in ("cov", "all"):
                nbytes += 8.0 * (2 * (nt - 1) * ns * ns + ns * ns + n * nd)
        if nrhs:
            nbytes += 8.0 * nnz + 16.0 * n * nrhs  # the factor; b and x
            flops += 4.0 * nnz * nrhs
    return {"bytes": nbytes, "flops": flops}


# ---- the same results in plain float64 torch ----------------------------------

def _exact(ns, nt, nd, blocks, b=None, want="diag"):
    """Block recursion on the blocks themselves: A = L L^T, then the selected
    inverse from Sigma L = L^{-T}."""
    D, B, C, corner = blocks
    T = torch.linalg.solve_triangular
    L, F, E = [], [], []  # L_ii, L_{i+1,i}, arrowhead row of L
    Sd = corner.clone()
    for i in range(nt):
        Di, Ci = D[i], C[i]
        if i:
            Di = Di - F[i - 1] @ F[i - 1].T
            Ci = Ci - E[i - 1] @ F[i - 1].T
        Li = torch.linalg.cholesky(Di)
        L.append(Li)
        if i < nt - 1:
            F.append(T(Li.T, B[i], upper=True, left=False))
        E.append(T(Li.T, Ci, upper=True, left=False))
        Sd = Sd - E[i] @ E[i].T
    Ld = torch.linalg.cholesky(Sd) if nd else Sd
    logdet = 2.0 * (sum(x.diagonal().log().sum() for x in L) + Ld.diagonal().log().sum())
    out = {"logdet": logdet.reshape(1).cpu().numpy()}
    if b is not None:
        r = torch.from_numpy(np.ascontiguousarray(b)).cuda()
        y, yd = [], r[nt * ns:].clone()
        for i in range(nt):
            ri = r[i * ns:(i + 1) * ns]
            if i:
                ri = ri - F[i - 1] @ y[i - 1]
            y.append(T(L[i], ri, upper=False))
            yd = yd - E[i] @ y[i]
        xd = T(Ld.T, T(Ld, yd, upper=False), upper=True) if nd else yd
        x = [None] * nt
        for i in reversed(range(nt)):
            yi = y[i] - E[i].T @ xd
            if i < nt - 1:
                yi = yi - F[i].T @ x[i + 1]
            x[i] = T(L[i].T, yi, upper=True)
        out["x"] = np.asfortranarray(torch.cat(x + [xd]).cpu().numpy())
    if want == "x":
        return {"x": out["x"]}

    def panel(i, d, f, e):  # one block column of the solver's layout, column-major
        return torch.cat(([d, f] if i < nt - 1 else [d]) + [e]).T.reshape(-1)

    if want == "all":
        cols = [panel(i, L[i], F[i] if i < nt - 1 else None, E[i]) for i in range(nt)]
        out["factor"] = torch.cat(cols + [Ld.T.reshape(-1)]).cpu().numpy()
    eye = torch.eye(ns, dtype=torch.float64, device="cuda")
    inv_d = T(Ld, torch.eye(nd, dtype=torch.float64, device="cuda"), upper=False) if nd else Ld
    Sdd = inv_d.T @ inv_d
    diag, cols = [Sdd.diagonal()], [Sdd.T.reshape(-1)]
    Sn = Sdn = None
    for i in reversed(range(nt)):
        inv = T(L[i], eye, upper=False)
        Y, W, Sf = Sdd @ E[i], inv, None
        if i < nt - 1:
            Sf = -(Sn @ F[i] + Sdn.T @ E[i]) @ inv
            Y = Y + Sdn @ F[i]
            W = W - F[i].T @ Sf
        Se = -Y @ inv
        Sn, Sdn = inv.T @ (W - E[i].T @ Se), Se
        diag.append(Sn.diagonal())
        if want == "cov":
            cols.append(panel(i, Sn, Sf, Se))
    out["diag"] = torch.cat(diag[::-1]).cpu().numpy()
    if want == "cov":
        out["cov"] = torch.cat(cols[::-1]).cpu().numpy()
    return out


def exact(case, seed):
    if case["kind"] == "batch":
        each = [_exact(*z, _blocks(*z, False, seed * 1009 + i))
                for i, z in enumerate(_batch_shapes(case))]
        return {"logdet": np.concatenate([e["logdet"] for e in each]),
                "diag": [e["diag"] for e in each]}
    ns, nt, nd = case["ns"], case["nt"], case["nd"]
    b = _rhs(ns * nt + nd, case["nrhs"], seed) if case["nrhs"] else None
    return _exact(ns, nt, nd, _blocks(ns, nt, nd, case["spde"], seed), b, case["want"])
