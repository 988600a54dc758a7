"""The work that the library's users have it do, as cases that can be timed.

A case names one public entry point, the problem it is called on and the
hierarchy's precision.  The problems are the package's own workloads
(chronoslab_b200.problems): the 7-point Laplacian, the Q1 elasticity cube and
the seeded log-normal diffusion, at sizes from a few thousand unknowns, where
a solve is a chain of short kernels, to nearly a million, where it streams the
operators from memory.  Every entry point gets what its caller holds before
the call: device vectors where it takes device pointers, host arrays where it
takes host arrays, and the handle of a finished setup where the program keeps
one.
"""
import ctypes
import math

import numpy as np
import torch

import chronoslab_b200 as cb
from chronoslab_b200 import problems as PB

PRECISION = {"fp32": cb.CHRONOS_FP32, "fp64": cb.CHRONOS_FP64}
ITMAX = 1000


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------

def listed():
    return [
        # one preconditioner application by a caller with its own Krylov loop,
        # on a small problem: launches and latency
        {"name": "vcycle_poisson_20_fp64", "kind": "vcycle", "problem": "poisson", "nx": 20,
         "precision": "fp64"},
        # the same on an ordinary size, FP32 vectors straight into an FP32 hierarchy
        {"name": "vcycle_elasticity_45_fp32", "kind": "vcycle", "problem": "elasticity", "nx": 45,
         "precision": "fp32"},
        # a small solve (the Poisson 32^3 workload of the benchmark)
        {"name": "pcg_poisson_32_fp32", "kind": "pcg", "problem": "poisson", "nx": 32,
         "precision": "fp32"},
        # an ordinary solve with the all-FP64 hierarchy
        {"name": "pcg_elasticity_24_fp64", "kind": "pcg", "problem": "elasticity", "nx": 24,
         "precision": "fp64"},
        # the large solve: the elasticity workload of the benchmark
        {"name": "pcg_elasticity_64_fp32", "kind": "pcg", "problem": "elasticity", "nx": 64,
         "precision": "fp32"},
        # a block of right-hand sides from host arrays (many load cases on one operator)
        {"name": "block_diffusion_64_x16_fp32", "kind": "block", "problem": "diffusion", "nx": 64,
         "nrhs": 16, "precision": "fp32"},
        # independent problems of uneven sizes solved together
        {"name": "batch_diffusion_12_fp32", "kind": "batch", "count": 12, "lo": 11, "hi": 40,
         "precision": "fp32"},
        # the backward direction: adjoint solve and gradient on the operator's pattern
        {"name": "adjoint_diffusion_48_fp64", "kind": "adjoint", "problem": "diffusion", "nx": 48,
         "precision": "fp64"},
        # the other Krylov callers (SQMR, GMRES), host vectors, at the size of the
        # reference's own regression problem
        {"name": "sqmr_elasticity_17_fp64", "kind": "sqmr", "problem": "elasticity", "nx": 17,
         "precision": "fp64"},
        # a setup from host arrays and the first application of its V-cycle
        {"name": "setup_diffusion_36_fp32", "kind": "setup", "problem": "diffusion", "nx": 36,
         "precision": "fp32"},
        # the FSAI numeric phase on device arrays, as a time stepper repeats it
        # when the operator's values change on a kept pattern
        {"name": "fsai_diffusion_61", "kind": "fsai", "problem": "diffusion", "nx": 61,
         "nstep": 15},
        # the Galerkin product of a caller with its own prolongation
        {"name": "galerkin_elasticity_26", "kind": "galerkin", "problem": "elasticity", "nx": 26},
    ]


def _size(rng, lo, hi):
    """A grid edge between lo and hi, spread over the logarithm of the unknowns."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["vcycle", "vcycle", "pcg", "pcg", "pcg", "block", "batch", "adjoint", "sqmr",
                       "gmres", "setup", "fsai", "galerkin"])
    case = {"kind": kind}
    if kind == "batch":
        case.update(count=rng.randint(3, 14), lo=rng.randint(9, 14), hi=rng.randint(18, 40))
    else:
        problem = rng.choice({"block": ["diffusion"], "adjoint": ["diffusion"],
                              "fsai": ["diffusion", "elasticity"],
                              "galerkin": ["diffusion", "elasticity"]}.get(
            kind, ["poisson", "elasticity", "elasticity", "diffusion"]))
        lo, hi = {"vcycle": (14, 72), "pcg": (14, 72), "block": (20, 64), "adjoint": (18, 56),
                  "sqmr": (14, 48), "gmres": (14, 48), "setup": (12, 36), "fsai": (20, 72),
                  "galerkin": (16, 60)}[kind]
        if problem == "elasticity":   # three unknowns per node and eleven times the entries per row
            lo, hi = max(8, lo // 2), {72: 60, 48: 24, 36: 18, 60: 28}[hi]
        case.update(problem=problem, nx=_size(rng, lo, hi))
    if kind == "block":
        case["nrhs"] = rng.randint(2, 16)
    if kind == "fsai":
        case["nstep"] = rng.choice([3, 8, 15, 24])
    elif kind != "galerkin":
        case["precision"] = rng.choice(["fp32", "fp32", "fp64"])
    return case


# ---------------------------------------------------------------------------
# The problems
# ---------------------------------------------------------------------------

def _elasticity(ne, modulus):
    """PB.elasticity_q1(ne, E=modulus) and the node coordinates, from the node
    stencils of a four-element cube: a node's 27 blocks depend only on which
    faces it lies on (and scale with modulus * h)."""
    small = PB.elasticity_q1(4)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    indptr, indices, data = small.indptr, small.indices, small.data
    table = np.zeros((3, 3, 3, 27, 3, 3))          # faces in x, y, z; offset; block
    for cz, z in enumerate((1, 2, 4)):              # next to the clamped face, inside, free face
        for cy, y in enumerate((0, 2, 4)):
            for cx, x in enumerate((0, 2, 4)):
                node = x + 5 * (y + 5 * (z - 1))
                for i in range(3):
                    for k in range(indptr[3 * node + i], indptr[3 * node + i + 1]):
                        c, j = divmod(int(indices[k]), 3)
                        dz, rem = divmod(c, 25)
                        dy, dx = divmod(rem, 5)
                        o = (dx - x + 1) + 3 * ((dy - y + 1) + 3 * (dz + 1 - z + 1))
                        table[cx, cy, cz, o, i, j] = data[k]
    table = torch.from_numpy(table * (4.0 * modulus / ne)).to(dev)
    m = ne + 1
    g = torch.arange(m * m * ne, device=dev)
    x, y, z = g % m, (g // m) % m, g // (m * m) + 1
    edge = lambda v: (v > 0).long() + (v == ne).long()             # noqa: E731
    cls = (edge(x), edge(y), (z > 1).long() + (z == ne).long())
    off = torch.arange(27, device=dev)
    ox, oy, oz = off % 3 - 1, (off // 3) % 3 - 1, off // 9 - 1
    cx, cy, cz = x[:, None] + ox, y[:, None] + oy, z[:, None] + oz
    ok = (cx >= 0) & (cx <= ne) & (cy >= 0) & (cy <= ne) & (cz >= 1) & (cz <= ne)
    node = cx + m * (cy + m * (cz - 1))
    n = 3 * g.numel()
    mask = ok[:, None, :, None].expand(-1, 3, 27, 3)
    vals = table[cls].permute(0, 2, 1, 3)[mask]
    cols = (3 * node[:, None, :, None] + torch.arange(3, device=dev)).expand(-1, 3, 27, 3)[mask]
    rowlen = (3 * ok.sum(1)).repeat_interleave(3)
    ptr = torch.zeros(n + 1, dtype=torch.int64, device=dev)
    ptr[1:] = torch.cumsum(rowlen, 0)
    A = type(small)((vals.cpu().numpy(), cols.int().cpu().numpy(), ptr.int().cpu().numpy()),
                    shape=(n, n))
    return A, (torch.stack([x, y, z], 1).double() / ne).cpu().numpy()


def _problem(case, seed, nx=None):
    """Operator (host CSR), test space and right-hand side of a case."""
    nx, seed = nx or case["nx"], seed + 1
    rng = np.random.default_rng(seed)
    name = case.get("problem", "diffusion")
    if name == "elasticity":
        A, X = _elasticity(nx, 0.9 + 0.2 * rng.random())
        return A, PB.rbm_test_space(X), PB.elasticity_rhs(A, X, seed)
    if name == "poisson":
        A = PB.poisson7(nx)
    else:
        A = PB.diffusion7(nx, seed=seed)[0]
    n = A.shape[0]
    b = PB.uniform_rhs(n, seed + 7, case.get("nrhs", 1))
    return A, np.ones((n, 1)), b


def _params(case, **more):
    if case.get("problem") != "elasticity":
        more["ntv"] = 1
    return cb.params(precision=PRECISION[case["precision"]], **more)


def _device(v, dtype=torch.float64):
    return torch.from_numpy(np.ascontiguousarray(v)).to("cuda", dtype)


def _vector_type(case):
    return torch.float32 if case["precision"] == "fp32" else torch.float64


def _batch_sizes(case):
    """The batch's grid edges, spread between its ends."""
    lo, hi, m = case["lo"], case["hi"], case["count"]
    return [int(round(lo * (hi / lo) ** (i / (m - 1)))) for i in range(m)]


def _fsai_inputs(case, seed):
    """An operator and the FSAI pattern found on an earlier one (another
    coefficient field or modulus) of the same grid."""
    G, ok = cb.fsai_pattern(_problem(case, 0)[0], nstep=case["nstep"], step_size=1, nthread=8,
                            fsai_fabs=1)
    assert ok
    return _problem(case, seed)[0], G


def _galerkin_inputs(case, seed):
    """An operator and the prolongation of an earlier one, as above."""
    A, TV, _ = _problem(case, 0)
    prm = cb.params(ntv=TV.shape[1])
    fc, _, S = cb.coarsen_device(A, prm)
    P, _ = cb.bamg(S, fc, np.linalg.qr(TV)[0], prm)
    P.sort_indices()
    return _problem(case, seed)[0], P


# ---------------------------------------------------------------------------
# prepare, run
# ---------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "fsai":
        A, G = _fsai_inputs(case, seed)
        s["n"] = A.shape[0]
        s["args"] = [_device(v, t) for v, t in (
            (A.indptr, torch.int32), (A.indices, torch.int32), (A.data, torch.float64),
            (G.indptr, torch.int32), (G.indices, torch.int32))]
        s["G"] = torch.zeros(G.nnz, dtype=torch.float64, device="cuda")
        return s
    if kind == "galerkin":
        s["A"], s["P"] = _galerkin_inputs(case, seed)
        return s
    if kind == "batch":
        probs = [_problem(case, 1000 * seed + i, nx) for i, nx in enumerate(_batch_sizes(case))]
        s["b"] = [p[2] for p in probs]
        s["h"] = cb.Batch([p[0] for p in probs], cb.params(
            precision=PRECISION[case["precision"]], ntv=1, nstep=15, step_size=4))
        return s
    A, TV, b = _problem(case, seed)
    if kind == "setup":
        s.update(A=A, TV=TV, prm=_params(case), precision=PRECISION[case["precision"]],
                 b=_device(b, _vector_type(case)))
        s["x"] = torch.zeros_like(s["b"])
        return s
    s["h"] = cb.Hierarchy(A, TV, _params(case))
    if kind == "vcycle":
        s.update(precision=PRECISION[case["precision"]], b=_device(b, _vector_type(case)))
        s["x"] = torch.zeros_like(s["b"])
    elif kind == "pcg":
        s["b"] = _device(b)
        s["x"] = torch.zeros_like(s["b"])
    elif kind == "adjoint":
        s["u"], s["g"] = np.random.default_rng(seed + 2).standard_normal(b.size), b
    else:                                  # block, sqmr, gmres: host arrays
        s["b"] = b
    return s


def run(s):
    kind = s["kind"]
    if kind == "vcycle":
        s["h"].vcycle_dev(s["b"].data_ptr(), s["x"].data_ptr(), s["precision"],
                          stream=torch.cuda.current_stream())
        return s["x"]
    if kind == "pcg":
        s["x"].zero_()
        it, flag, _ = s["h"].pcg_dev(s["b"].data_ptr(), s["x"].data_ptr(), ITMAX, 1e-8,
                                     stream=torch.cuda.current_stream())
        return {"x": s["x"], "iterations": it, "flag": flag}
    if kind == "block":
        x, its, flags, _ = s["h"].pcg_block(s["b"], itmax=ITMAX, tol=1e-8,
                                            stream=torch.cuda.current_stream())
        return {"x": x, "iterations": its, "flags": flags}
    if kind == "batch":
        xs, its, flags, _ = s["h"].solve(s["b"], ITMAX, 1e-8)
        return {"x": xs, "iterations": its, "flags": flags}
    if kind == "adjoint":
        lam, grad, it = s["h"].adjoint_grad(s["u"], s["g"], ITMAX, 1e-10)
        return {"lambda": lam, "grad": grad, "iterations": it}
    if kind == "sqmr":
        x, info, relres, it = cb.SQMR(s["h"], s["b"], 1e-6, 200)
        return {"x": x, "info": info, "iterations": it}
    if kind == "gmres":
        x, flag, relres, it, _ = cb.gmres_RIGHT(s["h"], s["b"], 50, 1e-6, 4)
        return {"x": x, "flag": flag, "iterations": list(it)}
    if kind == "setup":
        with cb.Hierarchy(s["A"], s["TV"], s["prm"]) as h:
            sizes = np.zeros(h.prm.nLevMax, np.int64)
            sizes[:h.nlevels] = [h.level_info(l)["n"] for l in range(h.nlevels)]
            h.vcycle_dev(s["b"].data_ptr(), s["x"].data_ptr(), s["precision"],
                         stream=torch.cuda.current_stream())
        return {"x": s["x"], "levels": sizes}
    if kind == "fsai":
        posdef = ctypes.c_int()
        ptr = [ctypes.c_void_p(t.data_ptr()) for t in s["args"]]
        cb.check(cb.load().chronos_fsai_numeric_noalloc(
            s["n"], *ptr, ctypes.c_void_p(s["G"].data_ptr()), ctypes.byref(posdef),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return {"G": s["G"], "posdef": posdef.value}
    C = cb.galerkin(s["A"], s["P"])
    return {"indptr": C.indptr, "indices": C.indices, "data": C.data}


# ---------------------------------------------------------------------------
# work: what a pass cannot do without
# ---------------------------------------------------------------------------

def _counts(case, nx=None):
    """Unknowns, operator entries and bytes per stored entry (values and a
    share of the column indices)."""
    nx = nx or case["nx"]
    vb = 4 if case.get("precision") == "fp32" else 8
    if case.get("problem") == "elasticity":
        m = nx + 1
        return 3 * m * m * nx, 9 * (3 * nx + 1) ** 2 * (3 * nx - 2), vb + 4 / 9
    return nx ** 3, 7 * nx ** 3 - 6 * nx ** 2, vb + 2


def _iterations(case, tol_digits):
    """About how many iterations the case's solve takes (iterations per digit
    from the benchmark's workloads; elasticity's grow with the mesh)."""
    nx, p = case.get("nx", 32), case.get("problem", "diffusion")
    per_digit = 2.4 if p == "poisson" else 5.5 if p == "diffusion" else 3.0 + 0.165 * nx
    return max(1.0, per_digit * tol_digits)


def _cycle(case, nx=None):
    """Bytes and operations of one V(1,1) cycle: the operator read for its two
    residuals (a third more on the coarse levels), the vectors once each."""
    n, nnz, eb = _counts(case, nx)
    vb = 4 if case.get("precision") == "fp32" else 8
    return 1.3 * (2 * nnz * eb) + 2 * n * vb, 1.3 * (4 * nnz + 24 * n)


def _solve(case, digits, nx=None, cols=1):
    """A preconditioned CG solve: per iteration a cycle, the operator once more
    and the five FP64 vectors of the recurrence read or written."""
    n, nnz, eb = _counts(case, nx)
    cyc_b, cyc_f = _cycle(case, nx)
    vec = 2 * n * (4 if case.get("precision") == "fp32" else 8)
    it = _iterations(case, digits)
    return {"bytes": it * (cyc_b - vec + nnz * eb + cols * (vec + 8 * 8 * n)),
            "flops": it * cols * (cyc_f + 2 * nnz + 12 * n)}


def work(case):
    kind = case["kind"]
    if kind == "batch":
        parts = [_solve(case, 8, nx) for nx in _batch_sizes(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    n, nnz, eb = _counts(case)
    if kind == "vcycle":
        b, f = _cycle(case)
        return {"bytes": b, "flops": f}
    if kind in ("pcg", "block"):
        return _solve(case, 8, cols=case.get("nrhs", 1))
    if kind == "adjoint":
        w = _solve(case, 10)
        return {"bytes": w["bytes"] + 8 * nnz, "flops": w["flops"] + nnz}
    if kind in ("sqmr", "gmres"):
        return _solve(case, 6)
    if kind == "setup":                    # read A once, write the hierarchy once
        return {"bytes": 3 * 12 * nnz, "flops": 60 * nnz}
    if kind == "fsai":                     # A and the pattern read, the values written
        k = min(1 + case["nstep"], 4 if case["problem"] != "elasticity" else 16)
        return {"bytes": 12 * nnz + n * k * 12, "flops": n * (k ** 3 / 3 + 2 * k * k)}
    return {"bytes": 12 * nnz + 12 * 4 * n + 12 * nnz / 8, "flops": 2 * 5 * nnz}


# ---------------------------------------------------------------------------
# exact: the same in plain torch, FP64
# ---------------------------------------------------------------------------

def _csr64(M):
    return torch.sparse_csr_tensor(torch.from_numpy(M.indptr.astype(np.int64)),
                                   torch.from_numpy(M.indices.astype(np.int64)),
                                   torch.from_numpy(np.asarray(M.data, np.float64)),
                                   size=M.shape, device="cuda")


def _cg(A, B):
    """Jacobi-preconditioned CG on every column of B, as far as FP64 goes."""
    M = _csr64(A)
    d = 1.0 / _device(A.diagonal())[:, None]
    B = _device(B if B.ndim == 2 else B[:, None])
    X, R = torch.zeros_like(B), B.clone()
    Z = d * R
    P, rz = Z.clone(), (R * Z).sum(0)
    norm = B.norm(dim=0).clamp_min(1e-300)
    for k in range(20000):
        Q = M @ P
        a = rz / (P * Q).sum(0).clamp_min(1e-300)
        X += a * P
        R -= a * Q
        if k % 50 == 49 and bool((R.norm(dim=0) < 2e-15 * norm).all()):
            break
        Z = d * R
        new = (R * Z).sum(0)
        P = Z + (new / rz.clamp_min(1e-300)) * P
        rz = new
    return X


def _vcycle64(h, b, l=0):
    """AMG_Vcycle with one FSAI pre- and post-smoothing step on the levels of a
    finished setup (its weights)."""
    A = h.export(l, "A")
    if l == h.nlevels - 1:
        return torch.linalg.solve(_device(A.toarray()), b)
    A, G, P = _csr64(A), h.export(l, "G"), h.export(l, "P")
    w, n, nc = h.level_info(l)["omega"], P.shape[0], P.shape[1]
    Gt, Pt = _csr64(G.T.tocsr()), _csr64(P.T.tocsr())
    G, P = _csr64(G), _csr64(P)
    x = w * (Gt @ (G @ b))
    x = x + P @ _vcycle64(h, Pt @ (b - A @ x), l + 1)
    return x + w * (Gt @ (G @ (b - A @ x)))


def _fsai64(A, G):
    """Row i of FSAI on G's pattern P + [i]: y = -A[P,P]^-1 A[P,i], scaled by
    1/sqrt(a_ii + A[i,P] y); rows of one length together."""
    n = A.shape[0]
    key = torch.repeat_interleave(torch.arange(n), torch.from_numpy(np.diff(A.indptr)).long()) * n
    key = (key + torch.from_numpy(A.indices).long()).cuda()
    val = _device(A.data)

    def entries(r, c):
        k = (r * n + c).reshape(-1)
        at = torch.searchsorted(key, k).clamp_max(key.numel() - 1)
        return torch.where(key[at] == k, val[at], 0.0).reshape(r.shape)

    ptr, ind = torch.from_numpy(G.indptr).long().cuda(), torch.from_numpy(G.indices).long().cuda()
    out = torch.zeros(ind.numel(), dtype=torch.float64, device="cuda")
    length = ptr[1:] - ptr[:-1]
    for m in torch.unique(length).tolist():
        for rows in torch.split(torch.nonzero(length == m).flatten(), 1 << 16):
            at = ptr[rows][:, None] + torch.arange(m, device="cuda")
            J = ind[at]                                      # m columns, the diagonal last
            S = entries(J[:, :, None].expand(-1, m, m), J[:, None, :].expand(-1, m, m))
            if m > 1:
                y = torch.linalg.solve(S[:, :-1, :-1], -S[:, :-1, -1:])[:, :, 0]
                scale = S[:, -1, -1] + (S[:, -1, :-1] * y).sum(1)
                row = torch.cat([y, torch.ones_like(y[:, :1])], 1)
            else:
                scale, row = S[:, 0, 0], torch.ones_like(S[:, 0])
            out[at] = row / torch.sqrt(scale)[:, None]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "fsai":
        return {"G": _fsai64(*_fsai_inputs(case, seed)), "posdef": None}
    if kind == "galerkin":
        A, P = _galerkin_inputs(case, seed)
        Pt, zero = P.T.tocsr(), np.longdouble(0)
        K = Pt @ (A @ P)                   # its pattern: entries that cancel exactly are dropped
        K.sort_indices()
        K.eliminate_zeros()
        C = (Pt.astype(np.longdouble) @ (A.astype(np.longdouble) @ P)).tocsr()
        C.sort_indices()
        nc = C.shape[0]
        key = np.repeat(np.arange(nc), np.diff(C.indptr)) * nc + C.indices
        want = np.repeat(np.arange(nc), np.diff(K.indptr)) * nc + K.indices
        at = np.minimum(np.searchsorted(key, want), key.size - 1)
        data = np.where(key[at] == want, C.data[at], zero).astype(np.float64)
        return {"indptr": None, "indices": None, "data": data}
    if kind == "batch":
        xs = []
        for i, nx in enumerate(_batch_sizes(case)):
            A, _, b = _problem(case, 1000 * seed + i, nx)
            xs.append(_cg(A, b)[:, 0])
        return {"x": xs, "iterations": None, "flags": None}
    A, TV, b = _problem(case, seed)
    if kind in ("vcycle", "setup"):
        with cb.Hierarchy(A, TV, _params(case)) as h:
            x = _vcycle64(h, _device(b, _vector_type(case)).double())
        return x if kind == "vcycle" else {"x": x, "levels": None}
    x = _cg(A, b)
    if kind == "block":
        return {"x": x, "iterations": None, "flags": None}
    x = x[:, 0]
    if kind == "adjoint":
        u = _device(np.random.default_rng(seed + 2).standard_normal(b.size))
        row = torch.repeat_interleave(torch.arange(A.shape[0]),
                                      torch.from_numpy(np.diff(A.indptr)).long()).cuda()
        grad = -x[row] * u[torch.from_numpy(A.indices).long().cuda()]
        return {"lambda": x, "grad": grad, "iterations": None}
    return {"x": x, **{k: None for k in (("iterations", "flag") if kind == "pcg" else
                                         ("info", "iterations"))}}
