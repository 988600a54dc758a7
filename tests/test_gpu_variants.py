"""Kernel variants at the edges of their ranges, against plain numpy."""
import numpy as np
import pytest
import scipy.sparse as sp

import chronoslab_b200 as cb

pytestmark = pytest.mark.gpu


def _banded_spd(n, band, seed):
    """Diagonally dominant SPD matrix with `band` sub-diagonals, some entries
    left out (the local systems then hold zeros)."""
    rng = np.random.default_rng(seed)
    A = sp.lil_matrix((n, n))
    for d in range(1, band + 1):
        v = rng.uniform(-1.0, 1.0, n - d) * (rng.random(n - d) < 0.7)
        A.setdiag(v, -d)
    A = sp.csr_matrix(A)
    A = A + A.T
    A = A + sp.diags(1.1 * np.asarray(abs(A).sum(1)).ravel() + 1.0)
    A = sp.csr_matrix(A)
    A.sort_indices()
    return A


@pytest.mark.parametrize("sizes", [[0, 1, 2, 3, 4], [4, 5, 7, 8], [8, 9, 15, 16], [16, 17, 31, 32],
                                   [32, 33, 63, 64], list(range(65))])
def test_fsai_local_systems_of_every_tile(lib, sizes):
    """Rows of G of the given local sizes, mixed within warps: each row equals
    y = -A[P,P]^-1 A[P,i] scaled by 1/sqrt(a_ii + A[i,P] y).  The local systems
    are diagonally dominant (condition below 50), so 64 unknowns give at most
    about 64 * 50 * 2.2e-16 = 7e-13 of the row's largest entry."""
    n = 400
    A = _banded_spd(n, 70, 5)
    rng = np.random.default_rng(1)
    rows, cols = [], []
    for i in range(n):
        m = min(sizes[int(rng.integers(len(sizes)))], i)
        P = np.sort(rng.choice(np.arange(max(0, i - 90), i), m, replace=False)) if m else []
        rows += [i] * (m + 1)
        cols += list(P) + [i]
    indptr = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))])
    G = sp.csr_matrix((np.ones(len(cols)), np.array(cols), indptr), shape=(n, n))
    vals, ok = cb.fsai_numeric(A, G)
    assert ok
    D = A.toarray()
    for i in range(n):
        c = G.indices[indptr[i]:indptr[i + 1]]
        P = c[:-1]
        y = -np.linalg.solve(D[np.ix_(P, P)], D[P, i])
        row = np.append(y, 1.0) / np.sqrt(D[i, i] + D[i, P] @ y)
        got = vals[indptr[i]:indptr[i + 1]]
        assert np.abs(got - row).max() <= 1e-12 * np.abs(row).max(), (i, len(P))


@pytest.mark.parametrize("m", [3, 8, 15, 16, 32, 40])
def test_fsai_indefinite_local_system(lib, m):
    """A local system with a negative pivot in its middle: is_posdef 0, that
    row the unit row, the others as if alone."""
    n = m + 90
    A = _banded_spd(n, 70, 9)
    bad = A.copy()
    k = m // 2
    bad[k, k] = -bad[k, k]
    bad = sp.csr_matrix(bad)
    bad.sort_indices()
    # rows before m diagonal only; row m takes all columns before it; the
    # rows after it the three before them
    cols = [[i] for i in range(m)] + [list(range(m + 1))]
    cols += [list(range(i - 3, i + 1)) if i - 3 > k else [i] for i in range(m + 1, n)]
    indptr = np.concatenate([[0], np.cumsum([len(c) for c in cols])])
    G = sp.csr_matrix((np.ones(indptr[-1]), np.concatenate(cols), indptr), shape=(n, n))
    good_vals, good = cb.fsai_numeric(A, G)
    vals, ok = cb.fsai_numeric(bad, G)
    assert good and not ok
    s, e = indptr[m], indptr[m + 1]
    assert np.array_equal(vals[s:e], np.append(np.zeros(m), 1.0))
    assert np.array_equal(vals[e:], good_vals[e:])


@pytest.mark.parametrize("nrhs", [1, 2, 3, 7, 8, 13, 16, 17])
def test_block_memory_orders_and_start_vectors(lib, nrhs):
    """Row-major, column-major and sliced blocks of right-hand sides give the
    same bits; started from its own solution a block stops at once."""
    from chronoslab_b200 import problems as PB
    A, _ = PB.diffusion7(15, seed=3)
    n = A.shape[0]
    B = np.ascontiguousarray(PB.uniform_rhs(n, 4, 18)[:, :nrhs])
    with cb.Hierarchy(A, np.ones(n), cb.params(ntv=1)) as h:
        X, its, flags, _ = h.pcg_block(B, tol=1e-8)
        assert X.shape == (n, nrhs) and np.all(flags == 0)
        assert np.all(np.linalg.norm(B - A @ X, axis=0) <= 1e-8 * np.linalg.norm(B, axis=0))
        wide = np.zeros((n, 2 * nrhs))
        wide[:, ::2] = B
        for other in (np.asfortranarray(B), wide[:, ::2]):
            X2, its2, _, _ = h.pcg_block(other, tol=1e-8)
            assert np.array_equal(X, X2) and np.array_equal(its, its2)
        # the block solve's recurrence starts from b - A x0 and always takes a step
        X3, its3, flags3, _ = h.pcg_block(B, X0=X, tol=1e-8)
        assert np.all(its3 == 1) and np.all(flags3 == 0)
        assert np.linalg.norm(X3 - X) <= 1e-6 * np.linalg.norm(X)


@pytest.mark.parametrize("nx", [4, 9, 22, 34])
@pytest.mark.parametrize("nrhs", [2, 5, 16])
def test_block_of_small_levels_matches_columns(lib, nx, nrhs):
    """Levels small enough that several lane sets share a row: each column
    solved to 1e-11 equals the column's own solve to 1e-8 (both residuals
    bounded, the operator's condition below 1e3 on these grids)."""
    from chronoslab_b200 import problems as PB
    A = PB.poisson7(nx)
    n = A.shape[0]
    B = PB.uniform_rhs(n, 9, nrhs)
    with cb.Hierarchy(A, np.ones(n), cb.params(ntv=1, maxCoarseSZ=20)) as h:
        X, its, flags, _ = h.pcg_block(B, tol=1e-11)
        assert np.all(flags == 0)
        for j in range(nrhs):
            x, it, _, flag, _ = h.pcg(B[:, j], tol=1e-11)
            assert flag == 0 and abs(int(its[j]) - it) <= 1
            assert np.linalg.norm(X[:, j] - x) <= 1e-8 * np.linalg.norm(x)


def _random_csr(m, n, lens, rng, lo=-1.0, hi=1.0):
    indptr = np.concatenate([[0], np.cumsum(lens)])
    idx = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lens]) if len(lens) else []
    return sp.csr_matrix((rng.uniform(lo, hi, indptr[-1]), np.asarray(idx, np.int64), indptr),
                         shape=(m, n))


@pytest.mark.parametrize("row_lens", [[0, 1, 2, 3], [5, 31, 32, 33, 64], [60, 130, 300],
                                      [1, 600, 2100], [2047, 2049, 3000]])
def test_galerkin_rows_of_every_table_size(lib, row_lens):
    """A = diagonal blocks coupling P's rows so that rows of the products fill
    the tables of every class and outgrow the largest: the same bits as a
    row-wise Gustavson product (scipy's, exact zeros dropped)."""
    rng = np.random.default_rng(len(row_lens) + sum(row_lens))
    n, nc = 160, 4000
    lens = rng.choice(row_lens, n)
    P = _random_csr(n, nc, lens, rng)
    P.data[rng.random(P.nnz) < 0.2] = 0.5          # exact cancellations against -0.5
    P.data[rng.random(P.nnz) < 0.2] = -0.5
    A = _random_csr(n, n, rng.integers(1, 7, n), rng)
    A.data[rng.random(A.nnz) < 0.3] = 1.0
    A = sp.csr_matrix(A + A.T)
    A.sort_indices()
    AP = sp.csr_matrix(A @ P)
    AP.eliminate_zeros()
    AP.sort_indices()
    want = sp.csr_matrix(sp.csr_matrix(P.T) @ AP)
    want.eliminate_zeros()
    want.sort_indices()
    got = cb.galerkin(A, P)
    assert np.array_equal(got.indptr, want.indptr)
    assert np.array_equal(got.indices, want.indices)
    assert np.array_equal(got.data, want.data)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 96, 97, 200, 257, 700])
def test_dense_cholesky_edges(lib, n):
    """Panels and tiles at their edges: |L L' - A| within 4 n eps |A| and the
    strict upper triangle zero; a negative pivot is refused wherever it lies."""
    rng = np.random.default_rng(n)
    B = rng.standard_normal((n, n))
    A = B @ B.T + n * np.eye(n)
    L = cb.dense_chol(A)
    assert not np.any(np.triu(L, 1))
    assert np.abs(L @ L.T - A).max() <= 4 * n * 2.2e-16 * np.abs(A).max()
    for k in {0, n // 2, n - 1}:
        C = A.copy()
        C[k, k] = -1.0
        with pytest.raises(cb.ChronosError) as e:
            cb.dense_chol(C)
        assert e.value.code == -4


@pytest.mark.parametrize("nx", [3, 4, 5, 7, 9])
def test_single_level_vcycle_is_the_dense_solve(lib, nx):
    """A problem no larger than the coarsest level: the V-cycle is A^-1 b, to
    the condition of the operator (below 200 here) times n eps."""
    from chronoslab_b200 import problems as PB
    A = PB.poisson7(nx)
    b = np.random.default_rng(nx).standard_normal(nx ** 3)
    with cb.Hierarchy(A, np.ones(nx ** 3), cb.params(precision=cb.CHRONOS_FP64, ntv=1)) as h:
        assert h.nlevels == 1
        x = h.vcycle(b)
    want = np.linalg.solve(A.toarray(), b)
    assert np.linalg.norm(x - want) <= 200 * nx ** 3 * 2.2e-16 * np.linalg.norm(want)


@pytest.mark.parametrize("prec,tol", [(cb.CHRONOS_FP64, 1e-12), (cb.CHRONOS_FP32, 2e-5)])
@pytest.mark.parametrize("problem,nx,coarse", [
    ("poisson", 11, 1000), ("poisson", 21, 50), ("poisson", 33, 1000), ("poisson", 50, 300),
    ("elasticity", 7, 100), ("elasticity", 11, 1000), ("elasticity", 18, 40),
    ("elasticity", 27, 300), ("fsai", 14, 200), ("fsai", 30, 1000)])
def test_folded_levels_match_the_operator_form(lib, problem, nx, coarse, prec, tol):
    """Every folded form (dense tails with even and odd rows, two, four and six
    kernels, wide restriction rows, smoother factors with long rows that stay
    unfolded) against the operator by operator cycle (spmv_format = 1), to the
    tolerances that the storage formats are held to; vectors in both types."""
    import torch
    from chronoslab_b200 import problems as PB
    if problem == "elasticity":
        A, X = PB.elasticity_q1(nx, return_coords=True)
        TV, more = PB.rbm_test_space(X), {}
    else:
        A = PB.poisson7(nx) if problem == "poisson" else PB.diffusion7(nx, seed=2)[0]
        TV, more = np.ones((A.shape[0], 1)), {"ntv": 1}
        if problem == "fsai":
            more.update(fsai_fabs=1)
    n = A.shape[0]
    b = np.random.default_rng(nx).standard_normal(n)
    with cb.Hierarchy(A, TV, cb.params(precision=prec, maxCoarseSZ=coarse, **more)) as hf, \
            cb.Hierarchy(A, TV, cb.params(precision=prec, maxCoarseSZ=coarse, spmv_format=1,
                                          **more)) as hp:
        assert hf.nlevels == hp.nlevels >= 2
        xf, xp = hf.vcycle(b), hp.vcycle(b)
        assert np.linalg.norm(xf - xp) <= tol * np.linalg.norm(xp)
        for t, code in ((torch.float32, cb.CHRONOS_FP32), (torch.float64, cb.CHRONOS_FP64)):
            bd = torch.from_numpy(b).to("cuda", t)
            out = torch.zeros_like(bd)
            hf.vcycle_dev(bd.data_ptr(), out.data_ptr(), code)
            torch.cuda.synchronize()
            got = out.double().cpu().numpy()
            assert np.linalg.norm(got - xp) <= max(tol, 2e-5 if t == torch.float32 else 0.0) \
                * np.linalg.norm(xp)
        x1, it1, _, f1, _ = hf.pcg(b, itmax=400, tol=1e-8)
        x2, it2, _, f2, _ = hp.pcg(b, itmax=400, tol=1e-8)
        assert f1 == 0 and f2 == 0 and abs(it1 - it2) <= 1
        assert np.linalg.norm(b - A @ x1) <= 1e-8 * np.linalg.norm(b)


@pytest.mark.parametrize("more", [{"precision": cb.CHRONOS_FP64}, {"precision": cb.CHRONOS_FP32},
                                  {"precision": cb.CHRONOS_FP32, "exact_outer": 1},
                                  {"precision": cb.CHRONOS_FP32, "replace_ratio": 0.5}])
def test_unrolled_loop_stops_as_the_host_loop(lib, more):
    """The device-side loop, several iterations per pass far from the tolerance,
    gives the one-iteration host loop's iterates bit for bit wherever a solve
    stops: at every itmax of a pass, at tolerances met inside one, at once."""
    from chronoslab_b200 import problems as PB
    A = PB.poisson7(14)
    n = A.shape[0]
    b = PB.uniform_rhs(n, 3)
    with cb.Hierarchy(A, np.ones(n), cb.params(ntv=1, maxCoarseSZ=100, **more)) as h1, \
            cb.Hierarchy(A, np.ones(n), cb.params(ntv=1, maxCoarseSZ=100, use_graph=0,
                                                  **more)) as h0:
        runs = [(k, 1e-12) for k in range(0, 11)] + [(100, 10.0 ** -e) for e in range(0, 13)]
        for itmax, tol in runs:
            x1, it1, rv1, f1, _ = h1.pcg(b, itmax=itmax, tol=tol)
            x0, it0, rv0, f0, _ = h0.pcg(b, itmax=itmax, tol=tol)
            assert (it1, f1) == (it0, f0), (itmax, tol)
            assert np.array_equal(x1, x0) and np.array_equal(rv1, rv0), (itmax, tol)
        bad = b.copy()
        bad[5] = np.nan
        with pytest.raises(cb.ChronosError):
            h1.pcg(bad)
        assert h1.pcg(b, tol=1e-8)[1] == h0.pcg(b, tol=1e-8)[1]


@pytest.mark.parametrize("prec", [cb.CHRONOS_FP64, cb.CHRONOS_FP32])
@pytest.mark.parametrize("nx,coarse", [(4, 1000), (9, 1000), (13, 100)])
def test_device_sqmr_loop(lib, nx, coarse, prec):
    """The device-side SQMR loop against the oracle's SQMR with the same V-cycle
    (iterations within one, solutions to the tolerance), the host loop bit for
    bit, with the operator passed in, at every small itmax, from the solution."""
    from chronoslab_b200 import problems as PB
    from oracle import amg_oracle as O
    A, X = PB.elasticity_q1(nx, return_coords=True)
    n, TV = A.shape[0], PB.rbm_test_space(X)
    b = np.random.default_rng(nx).standard_normal(n)
    prm = dict(precision=prec, maxCoarseSZ=coarse)
    with cb.Hierarchy(A, TV, cb.params(**prm)) as h, \
            cb.Hierarchy(A, TV, cb.params(use_graph=0, **prm)) as h0:
        x, info, relres, it = cb.SQMR(h, b, 1e-8, 200)
        assert info == 0
        assert relres == pytest.approx(np.linalg.norm(b - A @ x) / np.linalg.norm(b), rel=1e-6)
        xo, io, ro, ito, _ = O.sqmr(lambda v: A @ v, b, 1e-8, 200, lambda r: h.vcycle(r))
        assert io == 0 and abs(it - ito) <= 1
        assert np.linalg.norm(b - A @ x) <= 1.1e-8 * np.linalg.norm(b)
        xu, iu, _, itu = cb.SQMR(h, b, 1e-8, 200, A=A)
        assert iu == 0 and abs(itu - it) <= 1
        assert np.linalg.norm(xu - x) <= 1e-6 * np.linalg.norm(x)
        for itmax in (0, 1, 2, 5, it, it + 1):
            got, want = cb.SQMR(h, b, 1e-8, itmax), cb.SQMR(h0, b, 1e-8, itmax)
            assert np.array_equal(got[0], want[0]) and got[1:] == want[1:], itmax
            assert got[3] == min(itmax, it) and got[1] == (1 if itmax <= it else 0)
        # from the solution the first residual meets the test after one step
        x2, i2, _, it2 = cb.SQMR(h, b, 1e-6, 200, x0=x)
        assert i2 == 0 and it2 == 1


@pytest.mark.parametrize("prec", [cb.CHRONOS_FP64, cb.CHRONOS_FP32])
@pytest.mark.parametrize("lens", [[1], [2], [3], [1, 2, 4, 5], [7, 8, 9], [27], [1, 30, 64]])
def test_block_rows_of_every_length(lib, lens, prec):
    """The sliced 3x3 block form with odd, even, single and very uneven block
    rows that do not fill a chunk, against numpy: the first residual of a PCG
    from a random start (FP64 rows of at most 400 terms), and the solve, which a
    single-level hierarchy's exact preconditioner ends in two steps only if the
    outer product is A p."""
    rng = np.random.default_rng(sum(lens))
    nb = 301
    want = rng.choice(lens, nb)
    pat = sp.lil_matrix((nb, nb))
    for i in range(nb):
        pat[i, (i + rng.choice(nb, want[i] // 2, replace=False)) % nb] = 1.0
    pat = sp.csr_matrix(((pat + pat.T) > 0).astype(float))
    pat.setdiag(1.0)
    U = sp.csr_matrix(sp.kron(pat, np.ones((3, 3))))
    U.data = rng.uniform(-1.0, 1.0, U.nnz)
    A = sp.csr_matrix(U + U.T)                     # every block whole: nothing cancels
    A = sp.csr_matrix(A + sp.diags(np.asarray(abs(A).sum(1)).ravel() + 1.0))
    A.sort_indices()
    n = A.shape[0]
    b, x0 = rng.standard_normal(n), rng.standard_normal(n)
    with cb.Hierarchy(A, np.ones((n, 1)), cb.params(precision=prec, ntv=1, nLevMax=1)) as h:
        assert h.nlevels == 1 and h.level_info(0)["block_rows"] == nb
        x, it, rv, flag, _ = h.pcg(b, x0=x0, tol=1e-10, itmax=20)
        first = np.linalg.norm(b - A @ x0) / np.linalg.norm(b)
        assert rv[0] == pytest.approx(first, rel=1e-12)
        assert flag == 0 and it <= (2 if prec == cb.CHRONOS_FP64 else 3)
        assert np.linalg.norm(b - A @ x) <= 1e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("prec,io,tol", [(cb.CHRONOS_FP64, "float64", 1e-12),
                                         (cb.CHRONOS_FP32, "float64", 2e-5),
                                         (cb.CHRONOS_FP32, "float32", 2e-5)])
@pytest.mark.parametrize("shift", [0, 16])
def test_vcycle_in_place(lib, prec, io, tol, shift):
    """b and x the same device vector, or overlapping: the cycle of separate
    vectors up to the rounding of its forms."""
    import torch
    from chronoslab_b200 import problems as PB
    A = PB.poisson7(20)
    n = A.shape[0]
    ip = cb.CHRONOS_FP64 if io == "float64" else cb.CHRONOS_FP32
    with cb.Hierarchy(A, np.ones((n, 1)), cb.params(precision=prec, ntv=1)) as h:
        b = torch.from_numpy(np.random.default_rng(3).standard_normal(n)).to("cuda", getattr(torch, io))
        x = torch.empty_like(b)
        h.vcycle_dev(b.data_ptr(), x.data_ptr(), ip)
        both = torch.zeros(n + shift, dtype=b.dtype, device="cuda")
        both[:n] = b
        torch.cuda.synchronize()
        h.vcycle_dev(both.data_ptr(), both.data_ptr() + shift * both.element_size(), ip)
        torch.cuda.synchronize()
        err = (both[shift:].double() - x.double()).norm() / x.double().norm()
        assert float(err) <= tol


def test_free_while_a_caller_captures(lib):
    """A V-cycle in a caller's relaxed capture, during which another handle is
    destroyed: the capture survives and replays, and that handle's memory is
    given back by a later free."""
    import torch
    from chronoslab_b200 import problems as PB
    A = PB.poisson7(12)
    n = A.shape[0]
    prm = cb.params(precision=cb.CHRONOS_FP64, ntv=1)
    before = cb.device_bytes()
    with cb.Hierarchy(A, np.ones((n, 1)), prm) as h:
        other = cb.Hierarchy(A, np.ones((n, 1)), prm)
        b = torch.from_numpy(np.random.default_rng(3).standard_normal(n)).cuda()
        x = torch.zeros_like(b)
        h.vcycle_dev(b.data_ptr(), x.data_ptr())
        torch.cuda.synchronize()
        want = x.clone()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, capture_error_mode="relaxed"):
            h.vcycle_dev(b.data_ptr(), x.data_ptr(),
                         stream=torch.cuda.current_stream().cuda_stream)
            other.close()
        x.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(x, want)
        del g
        cb.Hierarchy(A, np.ones((n, 1)), prm).close()   # allocations and frees as before
    assert cb.device_bytes() == before


def test_folding_gives_way_to_the_memory_cap(lib, tmp_path):
    """Under the smallest CHRONOS_DEVICE_ALLOC_CAP (to 4 MB) at which a saved
    hierarchy of the same operators that is never folded (two presmoothing
    steps) loads, the foldable one loads and solves too (both from one warm
    autotuner cache: the same storage of the operators)."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    head = (f"import sys; sys.path.insert(0, {root!r})\n"
            "import numpy as np\nimport chronoslab_b200 as cb\n"
            "from chronoslab_b200 import problems as PB\nA = PB.poisson7(60)\nn = A.shape[0]\n")
    files = [str(tmp_path / f"pre{k}.chh") for k in (2, 1)]

    def child(code, cap=0):
        env = dict(os.environ, CHRONOS_TUNE_CACHE=str(tmp_path / "tune.txt"))
        if cap:
            env["CHRONOS_DEVICE_ALLOC_CAP"] = str(cap)
        r = subprocess.run([sys.executable, "-c", head + code], env=env, timeout=900,
                           capture_output=True, text=True)
        if r.returncode:
            assert cap and "ENOMEM" in r.stderr, r.stderr
            return None
        return [float(v) for v in r.stdout.split()[-2:]]

    lean, full = child(
        "out = []\n"
        f"for k, f in zip((2, 1), {files!r}):\n"
        "    with cb.Hierarchy(A, np.ones((n, 1)), cb.params(ntv=1, nupre=k,"
        " precision=cb.CHRONOS_FP64)) as h: h.save(f)\n"
        "    with cb.Hierarchy.load(f) as h: out.append(cb.device_bytes())\n"
        "print(*out)\n")
    assert full > lean
    solve = ("with cb.Hierarchy.load(%r) as h:\n"
             "    held = cb.device_bytes()\n    b = np.ones(n)\n"
             "    x, it, _, flag, _ = h.pcg(b, tol=1e-8, itmax=200)\n"
             "print(held, np.linalg.norm(b - A @ x) / np.linalg.norm(b))\n")
    low, high = int(lean), int(lean) + (512 << 20)
    assert child(solve % files[0], high)
    while high - low > 4 << 20:
        mid = (low + high) // 2
        if child(solve % files[0], mid):
            high = mid
        else:
            low = mid
    held, rel = child(solve % files[1], high)
    assert held < full and rel <= 1e-8


@pytest.mark.parametrize("first", [1, 31, 32, 33, 64, 65, 1000, 2430, 2500])
def test_dense_cholesky_names_the_first_bad_pivot(lib, first):
    """A matrix of many panel blocks with two non-positive pivots: refused with the
    first one's number (every block of a launch sees the same flag), and the next
    factorisation is untouched."""
    n = 2500
    rng = np.random.default_rng(first)
    A = np.diag(rng.uniform(1.0, 2.0, n))
    A[1:, 0] = A[0, 1:] = 0.01                       # diagonally dominant, L one full column
    bad = A.copy()
    for k in {first, min(first + 40, n)}:
        bad[k - 1, k - 1] = -1.0
    with pytest.raises(cb.ChronosError, match=f"pivot {first}$") as e:
        cb.dense_chol(bad)
    assert e.value.code == -4
    L = cb.dense_chol(A)
    assert np.abs(L @ L.T - A).max() <= 4 * n * 2.2e-16 * np.abs(A).max()


@pytest.mark.parametrize("first", [8, 101, 108])
@pytest.mark.parametrize("second", [1, 8, 108])
def test_second_tuning_of_the_finest_operator(lib, tmp_path, first, second):
    """FP32 hierarchy with the exact outer product: the finest operator's storage is
    chosen twice, for FP32 and for FP64 (the decisions set here: lanes, + 100 for
    sliced ELL, which leaves rows above 32 entries to whole warps).  Whatever is
    chosen, the cycle is the FP64 hierarchy's to FP32 rounding and the solve
    converges."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    A = _poisson_with_long_rows()
    longest = int(np.diff(A.indptr).max())
    assert longest > 32 and A.nnz <= 16 * A.shape[0]
    tune = tmp_path / "tune.txt"
    tune.write_text("".join(
        f"v2 {kind} {A.shape[0]} {A.nnz} {A.shape[1]} {fp32} {longest} {first if fp32 else second}\n"
        for kind in "hH" for fp32 in (0, 1)))
    sp.save_npz(tmp_path / "A.npz", A)
    code = (f"import sys; sys.path.insert(0, {root!r})\n"
            "import numpy as np, scipy.sparse as sp\nimport chronoslab_b200 as cb\n"
            f"A = sp.csr_matrix(sp.load_npz({str(tmp_path / 'A.npz')!r}))\nn = A.shape[0]\n"
            "b = np.random.default_rng(1).standard_normal(n)\n"
            "prm = dict(ntv=1, nupre=2, maxCoarseSZ=200)\n"
            "with cb.Hierarchy(A, np.ones((n, 1)), cb.params(precision=cb.CHRONOS_FP32,"
            " exact_outer=1, **prm)) as h, cb.Hierarchy(A, np.ones((n, 1)),"
            " cb.params(precision=cb.CHRONOS_FP64, spmv_format=1, **prm)) as h64:\n"
            "    x, y = h.vcycle(b), h64.vcycle(b)\n"
            "    z, it, _, flag, _ = h.pcg(b, tol=1e-8)\n"
            "print(np.linalg.norm(x - y) / np.linalg.norm(y),"
            " np.linalg.norm(b - A @ z) / np.linalg.norm(b), flag)\n")
    r = subprocess.run([sys.executable, "-c", code], env=dict(os.environ, CHRONOS_TUNE_CACHE=str(tune)),
                       timeout=600, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    err, res, flag = [float(v) for v in r.stdout.split()]
    assert err <= 2e-5 and res <= 1e-8 and flag == 0


def _poisson_with_long_rows():
    """poisson7(14) with five rows of 60 further weak couplings."""
    from chronoslab_b200 import problems as PB
    A = sp.lil_matrix(PB.poisson7(14))
    rng = np.random.default_rng(8)
    for i in (3, 700, 1301, 2000, 2743):
        for j in rng.choice(2744, 60, replace=False):
            if i != j:
                A[i, j] = A[j, i] = -0.01
    A = sp.csr_matrix(A)
    A = sp.csr_matrix(A + sp.identity(2744))
    A.sort_indices()
    return A


@pytest.mark.parametrize("prec", [cb.CHRONOS_FP64, cb.CHRONOS_FP32])
@pytest.mark.parametrize("problem", ["identity", "poisson"])
@pytest.mark.parametrize("tol", [0.0, -1.0, np.nan, np.inf])
def test_loops_agree_at_odd_tolerances(lib, prec, problem, tol):
    """A tolerance that no residual meets, or every one, and a residual that becomes
    exactly zero (a multiple of the identity, whose inverse is exact): the device-side
    loop ends where the one-iteration host loop ends, in the same way."""
    from chronoslab_b200 import problems as PB
    A = PB.poisson7(8) if problem == "poisson" else sp.csr_matrix(2.0 * sp.identity(64))
    n = A.shape[0]
    b = np.arange(1.0, n + 1.0)
    out = []
    for use_graph in (1, 0):
        with cb.Hierarchy(A, np.ones((n, 1)), cb.params(
                precision=prec, ntv=1, use_graph=use_graph, maxCoarseSZ=100)) as h:
            for itmax in (1, 3, 9):
                try:
                    x, it, rv, flag, _ = h.pcg(b, itmax=itmax, tol=tol)
                    out.append((x.tobytes(), it, rv.tobytes(), flag))
                except cb.ChronosError as e:
                    out.append(str(e))
    assert out[:3] == out[3:]


def _with_hub(nx, reach):
    """poisson7(nx) and one node before it, coupled to the first `reach` nodes."""
    from chronoslab_b200 import problems as PB
    m = nx ** 3
    c = np.zeros(m)
    c[:reach] = -0.5
    A = sp.bmat([[sp.csr_matrix([[0.5 * reach + 2.0]]), sp.csr_matrix(c)],
                 [sp.csr_matrix(c[:, None]), PB.poisson7(nx) + sp.identity(m)]], format="csr")
    A.sort_indices()
    return A


@pytest.mark.parametrize("prec,tol", [(cb.CHRONOS_FP64, 1e-12), (cb.CHRONOS_FP32, 2e-5)])
@pytest.mark.parametrize("nx,reach", [(11, 1331), (13, 2197), (20, 500), (20, 2040), (20, 2050),
                                      (30, 27000), (40, 1500)])
def test_folded_levels_with_a_hub_row(lib, nx, reach, prec, tol):
    """One row of the smoother with up to all columns (below, at and above what the
    two-matrix apply takes): the operator form's cycle, and the same iterations."""
    A = _with_hub(nx, reach)
    n = A.shape[0]
    b = np.random.default_rng(nx).standard_normal(n)
    prm = dict(precision=prec, ntv=1, maxCoarseSZ=400)
    with cb.Hierarchy(A, np.ones((n, 1)), cb.params(**prm)) as hf, \
            cb.Hierarchy(A, np.ones((n, 1)), cb.params(spmv_format=1, **prm)) as hp:
        xf, xp = hf.vcycle(b), hp.vcycle(b)
        assert np.linalg.norm(xf - xp) <= tol * np.linalg.norm(xp)
        r1, r2 = hf.pcg(b, tol=1e-8), hp.pcg(b, tol=1e-8)
        assert r1[3] == r2[3] == 0 and abs(r1[1] - r2[1]) <= 1


def test_hub_row_does_not_fill_the_setup(lib):
    """39,305 rows, one coupled to all others: A S would have 1.5e9 entries, which no
    fold keeps.  Folding and tuning take no longer than the rest of the setup."""
    A = _with_hub(34, 34 ** 3)
    with cb.Hierarchy(A, np.ones((A.shape[0], 1)), cb.params(
            precision=cb.CHRONOS_FP64, ntv=1)) as h:
        t = h.setup_times()
    with cb.Hierarchy(A, np.ones((A.shape[0], 1)), cb.params(
            precision=cb.CHRONOS_FP64, ntv=1)) as h:
        t = h.setup_times()
    assert t["autotune"] <= t["total"] - t["autotune"]


@pytest.mark.parametrize("nrhs", [1, 2, 5, 16])
@pytest.mark.parametrize("prec", [cb.CHRONOS_FP64, cb.CHRONOS_FP32])
def test_single_level_block(lib, nrhs, prec):
    """A problem that is its own coarsest level, with a condition of 1e12: the inverse
    is good to a few digits and a solve takes several steps.  Each column takes the
    steps of its own solve, whatever the memory of the block's scalars held before
    (not-a-numbers here)."""
    n = 120
    Q, _ = np.linalg.qr(np.random.default_rng(2).standard_normal((n, n)))
    D = (Q * np.logspace(-12, 0, n)) @ Q.T
    A = sp.csr_matrix(0.5 * (D + D.T))
    B = A @ np.random.default_rng(3).standard_normal((n, nrhs))
    with cb.Hierarchy(A, np.ones((n, 1)), cb.params(precision=prec, ntv=1, exact_outer=1)) as h:
        assert h.nlevels == 1
        single = [h.pcg(np.ascontiguousarray(B[:, j]), itmax=40, tol=1e-14) for j in range(nrhs)]
        for k in 3 * list(range(3, 40)):
            with pytest.raises(cb.ChronosError):
                cb.dense_chol(np.full((k, k), np.nan))
        X, its, flags, _ = h.pcg_block(B, itmax=40, tol=1e-14)
        for j in range(nrhs):
            _, it, rv, flag, _ = single[j]
            assert flag == flags[j] == 0 and it >= 2 and abs(int(its[j]) - it) <= 1, (it, its[j])


@pytest.mark.parametrize("nrhs", [3, 16, 17, 35])
def test_row_major_blocks_of_any_width(lib, nrhs):
    """chronos_pcg_block_rows on row-major right-hand sides, wider than one solve's 16
    columns too (rows then lie apart), with and without start vectors: the bits of the
    column-major call."""
    import ctypes as C
    from chronoslab_b200 import problems as PB
    A = PB.poisson7(11)
    n = A.shape[0]
    rng = np.random.default_rng(nrhs)
    B, X0 = rng.standard_normal((n, nrhs)), rng.standard_normal((nrhs, n))
    pd, pi = C.POINTER(C.c_double), C.POINTER(C.c_int)

    def solve(h, b, rows, x0):
        x, its, fl = np.full((nrhs, n), 7.0), np.zeros(nrhs, np.int32), np.ones(nrhs, np.int32)
        cb.check(lib.chronos_pcg_block_rows(
            h._h, nrhs, b.ctypes.data_as(pd), rows, None if x0 is None else x0.ctypes.data_as(pd),
            x.ctypes.data_as(pd), 200, 1e-8, its.ctypes.data_as(pi), fl.ctypes.data_as(pi), None,
            None))
        assert not fl.any()
        return x, its

    with cb.Hierarchy(A, np.ones((n, 1)), cb.params(ntv=1, maxCoarseSZ=100)) as h:
        for x0 in (None, X0):
            by_rows = solve(h, np.ascontiguousarray(B), 1, x0)
            by_cols = solve(h, np.ascontiguousarray(B.T), 0, x0)
            assert np.array_equal(by_rows[0], by_cols[0]) and np.array_equal(by_rows[1], by_cols[1])
            assert np.all(np.linalg.norm(B - A @ by_rows[0].T, axis=0)
                          <= 1e-8 * np.linalg.norm(B, axis=0))
