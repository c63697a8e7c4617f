"""The FP64 CG kernel (ILLT by FP64 Jacobi sweeps, or the identity) on caller matrices of the sizes where its
row split changes: fewer rows than a CTA's minimum, partial last CTAs, one row more than the CTAs hold, and
a system whose vectors do not fit shared memory."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from nonlocal_gb300 import _lib
    from nonlocal_gb300 import thermal as T
    if _lib.device_count() == 0:
        pytest.skip("no CUDA device")
    return T.Context()


def banded(n, band, seed, dominance):
    """A symmetric matrix of `band` random off-diagonals (every third one empty beyond the first) whose diagonal is
    `dominance` times the row's absolute sum: eigenvalues within (1 -+ 1 / dominance) of the diagonal."""
    import scipy.sparse as sp
    rng = np.random.default_rng(seed)
    offs = [k for k in range(1, band + 1) if k < n and (k == 1 or k % 3)]
    U = sp.diags([-rng.uniform(0.1, 1.0, n - k) for k in offs], offs, shape=(n, n)) if offs else sp.csr_matrix((n, n))
    A = (U + U.T).tocsr()
    d = dominance * np.maximum(np.asarray(abs(A).sum(axis=1)).ravel(), 1.0)
    return (A + sp.diags(d)).tocsr(), (U + sp.diags(d)).tocsr()


@pytest.mark.parametrize("preconditioned", [True, False])
@pytest.mark.parametrize("n, band", [(1, 1), (7, 3), (8, 2), (9, 8), (33, 40), (152 * 8, 5), (152 * 8 + 1, 17),
                                     (152 * 16 - 3, 30), (5003, 70), (152 * 1024 + 5, 4)])
def test_pcg_sizes(ctx, n, band, preconditioned):
    from scipy.sparse.linalg import spsolve
    from nonlocal_gb300 import thermal as T
    A, U = banded(n, band, n, 1.25)
    U.sort_indices()
    csr = (U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data)
    b = np.random.default_rng(1).standard_normal(n)
    x, rep = T.conjugate_gradient(ctx, csr, b, preconditioner_csr=csr if preconditioned else None, tolerance=1e-12)
    assert np.linalg.norm(b - A @ x) <= 1.01e-12 * np.linalg.norm(b)
    assert rep.residual <= 1e-12
    # |x - x*| <= |r| / lambda_min, lambda_min >= 0.2 / 1.25 of the smallest diagonal
    ref = spsolve(A.tocsc(), b)
    lo = A.diagonal().min() * 0.2 / 1.25
    assert np.linalg.norm(x - ref) <= 2e-12 * np.linalg.norm(b) / lo
    # from the solution itself: nothing left to do
    again, rep2 = T.conjugate_gradient(ctx, csr, b, x0=x, preconditioner_csr=csr if preconditioned else None,
                                       tolerance=1e-11)
    assert rep2.iterations == 0 and np.array_equal(again, x)


def test_slowly_contracting_factor_takes_the_exact_sweeps(ctx):
    """A tridiagonal matrix: IC(0) is the exact factor, whose Jacobi sweeps would need hundreds of steps, so the
    solve goes back to the exact triangular sweeps and ends after one or two iterations."""
    from nonlocal_gb300 import thermal as T
    n = 700
    rp = np.append(np.arange(0, 2 * n, 2), 2 * n - 1).astype(np.int64)
    col = np.empty(2 * n - 1, dtype=np.int64)
    val = np.empty(2 * n - 1)
    col[0::2], col[1::2] = np.arange(n), np.arange(1, n)
    val[0::2], val[1::2] = 2.0001, -1.0
    b = np.sin(0.37 * np.arange(n))
    x, rep = T.conjugate_gradient(ctx, (rp, col, val), b, preconditioner_csr=(rp, col, val), tolerance=1e-10)
    assert rep.iterations <= 3 and rep.residual <= 1e-10
    r = b - 2.0001 * x
    r[:-1] += x[1:]
    r[1:] += x[:-1]
    assert np.linalg.norm(r) <= 1.01e-10 * np.linalg.norm(b)


def test_caller_rows_in_any_order(ctx):
    """The caller's upper rows unsorted, with entries given in two parts, rows without a diagonal, the arrays starting
    at an offset: the solve is that of the same matrix sorted and summed; a column below the diagonal or out of range
    is refused."""
    import scipy.sparse as sp
    from nonlocal_gb300 import _lib
    from nonlocal_gb300 import thermal as T
    rng = np.random.default_rng(7)
    n = 301
    A, U = banded(n, 45, 3, 1.25)
    U = U.tocoo()
    r, c, v = U.row, U.col, U.data
    split = rng.random(r.size) < 0.2                       # a fifth of the entries in two parts
    r, c, v = np.concatenate([r, r[split]]), np.concatenate([c, c[split]]), np.concatenate([v, 0.25 * v[split]])
    v[:split.size][split] *= 0.75
    order = rng.permutation(r.size)
    order = order[np.argsort(r[order], kind="stable")]     # by row, any order inside
    off = 5
    rp = off + np.concatenate([[0], np.cumsum(np.bincount(r, minlength=n))]).astype(np.int64)
    col = np.concatenate([np.full(off, -9), c[order]]).astype(np.int64)
    val = np.concatenate([np.full(off, np.nan), v[order]])
    b = rng.standard_normal(n)
    x, rep = T.conjugate_gradient(ctx, (rp, col, val), b, tolerance=1e-12)
    assert rep.nnz_solver == sum((k + 3) // 4 * 4 for k in np.bincount(r, minlength=n) + np.bincount(c[r != c], minlength=n))
    assert np.linalg.norm(b - A @ x) <= 1.01e-12 * np.linalg.norm(b)
    for wrong in (0, n):
        bad = col.copy()
        bad[rp[n - 1]] = wrong
        with pytest.raises(_lib.NlgpuError):
            T.conjugate_gradient(ctx, (rp, bad, val), b)


@pytest.mark.parametrize("n, band", [(1, 1), (31, 3), (64, 2), (65, 70), (152 * 64, 5), (152 * 64 + 1, 9), (152 * 96 + 40, 33),
                                     (400001, 3)])
def test_jacobi_application_sizes(ctx, n, band):
    """The FP32 ILLT application at the edges of its row split (and past the size of the one-launch form): on a
    strongly dominant matrix a sweep contracts by at least 2.5, so 24 sweeps per triangle are the exact application to FP32
    rounding, and 32 and 33 sweeps (one launch, one per sweep) agree."""
    from nonlocal_gb300 import thermal as T
    _, U = banded(n, band, 11, 4.0)
    U.sort_indices()
    pre = T.EigenILLTPreconditioner(ctx)
    assert pre.compute((U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data)).computation_info() == pre.SUCCESS
    x = np.random.default_rng(2).standard_normal(n)
    exact = pre.solve(x)
    # an entry's sum has at most `band` terms of FP32 products, twice; the sweeps' remainder is 2.5^-24
    tol = (2 * (band + 4) * np.finfo(np.float32).eps + 2.5 ** -24) * np.abs(exact).max()
    for sweeps in (24, 32, 33):
        assert np.abs(pre.solve_f32(x, sweeps) - exact).max() <= tol, sweeps


def test_large_identity_systems_go_by_launches():
    """34 million entries and more: a launch per phase, so several an iteration; fewer: one kernel for them all."""
    from nonlocal_gb300 import _lib
    from nonlocal_gb300 import thermal as T
    from nonlocal_gb300.meshgen import structured_quad_mesh
    if _lib.device_count() == 0:
        pytest.skip("no CUDA device")
    mesh = structured_quad_mesh(200, 150, "bilinear")
    for radius, large in ((0.05, False), (0.13, True)):
        pb = T.Problem2D.from_mesh(mesh)
        pb.set_model(T.Model2D(influence="fast_polynomial", radius=(radius, radius), local_weight=0.5))
        pb.add_boundary(T.Boundary(edges=mesh.boundaries["left"], kind="temperature", value=1.0))
        pb.add_boundary(T.Boundary(edges=mesh.boundaries["right"], kind="flux", value=0.7))
        pb.find_neighbours()
        pb.conductivity_matrix("FULL")
        before = _lib.kernel_launches()
        x, rep = pb.solve_assembled(tolerance=1e-11, preconditioner="identity")
        launches = _lib.kernel_launches() - before
        assert (rep.nnz_solver > 2 ** 25) == large
        assert launches >= 5 * rep.iterations if large else launches < rep.iterations
        assert rep.residual <= 1e-11
        y, ref = pb.solve_assembled(tolerance=1e-11)   # ILLT
        # both residuals at most 1e-11 |b|; |A^-1| |b| / |x| <= the condition number, below 1e6 here
        assert np.linalg.norm(x - y) <= 2e-5 * np.linalg.norm(y)
        with pytest.raises(_lib.NlgpuError) as e:   # the limit of iterations
            pb.solve_assembled(tolerance=1e-11, preconditioner="identity", max_iterations=1)
        assert e.value.status == 6


def arrow(n, dense):
    """A diagonally dominant arrow: the rows in `dense` hold every column (eigenvalues 1 to 3 times the diagonal's
    smallest by Gershgorin's circles)."""
    import scipy.sparse as sp
    rng = np.random.default_rng(n)
    rows = [sp.csr_matrix((rng.uniform(-1.0, 1.0, n - 1 - r), (np.full(n - 1 - r, r), np.arange(r + 1, n))), shape=(n, n))
            for r in dense]
    U = sum(rows[1:], rows[0])
    A = (U + U.T).tocsr()
    d = 2.0 * np.maximum(np.asarray(abs(A).sum(axis=1)).ravel(), 1.0)
    return (A + sp.diags(d)).tocsr(), (U + sp.diags(d)).tocsr()


@pytest.mark.parametrize("n, dense", [(255, [0]), (256, [0]), (257, [0, 3]), (513, [5]), (1025, [0, 1]),
                                      (5000, [0, 2500, 4000]), (20011, [7])])
def test_dense_rows(ctx, n, dense):
    """Rows as long as the matrix: at the lengths where runs are merged, columns and rows of the full matrix."""
    from nonlocal_gb300 import thermal as T
    A, U = arrow(n, dense)
    U.sort_indices()
    csr = (U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data)
    b = np.random.default_rng(2).standard_normal(n)
    x, rep = T.conjugate_gradient(ctx, csr, b, tolerance=1e-12)
    assert np.linalg.norm(b - A @ x) <= 1.01e-12 * np.linalg.norm(b)
    again, _ = T.conjugate_gradient(ctx, csr, b, tolerance=1e-12)
    assert np.array_equal(again, x)


@pytest.mark.parametrize("n", [120000, 3000000])
def test_a_dense_row_costs_no_more_than_its_entries(ctx, n):
    """All columns in one row: its sort and its products take milliseconds.  (With 120 000 columns ranking the row
    took 10 s, the host's sort and the products 15 ms; with 3 million its products by a few lanes took 2 s.)"""
    import time
    from nonlocal_gb300 import thermal as T
    A, U = arrow(n, [0])
    U.sort_indices()
    csr = (U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data)
    b = np.random.default_rng(2).standard_normal(n)
    T.conjugate_gradient(ctx, csr, b, tolerance=1e-10)
    t0 = time.perf_counter()
    x, rep = T.conjugate_gradient(ctx, csr, b, tolerance=1e-10)
    assert time.perf_counter() - t0 < 1.0
    assert np.linalg.norm(b - A @ x) <= 1.01e-10 * np.linalg.norm(b)


@pytest.mark.parametrize("n", [40, 700])
def test_split_entries_are_added_in_one_order(ctx, n):
    """Entries split into parts of very different size (equal columns in the caller's order): the same bits on every call."""
    from nonlocal_gb300 import thermal as T
    rng = np.random.default_rng(n)
    rp, col, val = [0], [], []
    for r in range(n):
        cols = np.sort(rng.integers(r, n, 12))
        cols[0] = r
        col += [r] + cols.tolist()
        val += [60.0] + (rng.standard_normal(12) * 10.0 ** rng.integers(-8, 1, 12)).tolist()
        rp.append(len(col))
    csr = (np.array(rp), np.array(col), np.array(val))
    b = rng.standard_normal(n)
    first, _ = T.conjugate_gradient(ctx, csr, b, tolerance=1e-12)
    for _ in range(12):
        assert np.array_equal(T.conjugate_gradient(ctx, csr, b, tolerance=1e-12)[0], first)


@pytest.mark.parametrize("blocks", [1, 50, 5000])
def test_pivots_that_fail_take_the_exact_factor(ctx, blocks):
    """Kershaw's matrix, positive definite, whose IC(0) has a negative pivot: the fixed-point sweeps fail, and the exact
    factorisation retries with its diagonal shifts."""
    import scipy.sparse as sp
    from nonlocal_gb300 import thermal as T
    K = np.array([[3.0, -2, 0, 2], [-2, 3, -2, 0], [0, -2, 3, -2], [2, 0, -2, 3]])
    A = sp.kron(sp.identity(blocks), K).tocsr()
    U = sp.triu(A).tocsr()
    U.eliminate_zeros()
    U.sort_indices()
    csr = (U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data)
    b = np.random.default_rng(0).standard_normal(4 * blocks)
    x, rep = T.conjugate_gradient(ctx, csr, b, preconditioner_csr=csr, tolerance=1e-11)
    assert rep.preconditioner_ok and rep.preconditioner_shifts >= 1
    assert np.linalg.norm(b - A @ x) <= 1.01e-11 * np.linalg.norm(b)
