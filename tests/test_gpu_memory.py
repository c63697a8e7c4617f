"""Buffers that are kept and handed on: contexts made and destroyed in turn, problems of changing size on one
context, and several threads at once, each against the direct solution."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    from nonlocal_gb300 import _lib
    from nonlocal_gb300 import thermal
    if _lib.device_count() == 0:
        pytest.skip("no CUDA device")
    return thermal


SIZES = [1, 40, 700, 3000, 41, 699, 90000, 2]


def check(T, ctx, n, seed):
    """A diagonally dominant tridiagonal system (eigenvalues within 3 / 5 of the diagonal 5): the error is at most
    the residual / 2, the residual at most the tolerance * |b|."""
    import scipy.sparse as sp
    from scipy.sparse.linalg import spsolve
    rng = np.random.default_rng(seed)
    off = [rng.uniform(-1.0, 1.0, n - k) for k in (1,) if n > k]
    U = sp.diags([np.full(n, 5.0)] + off, range(1 + len(off)), shape=(n, n)).tocsr()
    A = (U + U.T - sp.diags(U.diagonal())).tocsr()
    b = rng.standard_normal(n)
    csr = (U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data)
    x, rep = T.conjugate_gradient(ctx, csr, b, preconditioner_csr=csr if seed % 2 else None, tolerance=1e-12)
    assert rep.residual <= 1e-12
    return np.linalg.norm(x - spsolve(A.tocsc(), b)) <= 1.01e-12 * np.linalg.norm(b)


def test_sizes_in_turn_on_one_context(T):
    ctx = T.Context()
    assert all(check(T, ctx, n, k) for k, n in enumerate(SIZES * 2))


def test_contexts_in_turn(T):
    for k, n in enumerate(SIZES * 2):
        assert check(T, T.Context(), n, k)


def test_threads(T):
    bad = []

    def work(seed):
        try:
            for k, n in enumerate((SIZES[seed:] + SIZES[:seed]) * 6):
                if not check(T, T.Context(), n, seed + k):
                    bad.append((seed, n))
        except Exception as e:   # reported by the main thread
            bad.append((seed, repr(e)))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_idle_memory_is_bounded_and_given_back(T):
    """Sixteen contexts whose last call left several hundred megabytes each: at most 4 GiB stay idle, and go back when
    asked for, with the contexts alive and after them; the contexts work on."""
    import torch
    free = lambda: torch.cuda.mem_get_info()[0]
    torch.cuda.init()
    contexts = [T.Context() for _ in range(16)]
    T.release_idle_memory()
    n = 1500000
    csr = (np.append(np.arange(0, 2 * n, 2), 2 * n - 1), np.empty(2 * n - 1, dtype=np.int64), np.empty(2 * n - 1))
    csr[1][0::2], csr[1][1::2] = np.arange(n), np.arange(1, n)
    csr[2][0::2], csr[2][1::2] = 5.0, -1.0
    b = np.ones(n)
    x = [T.conjugate_gradient(c, csr, b, preconditioner_csr=csr, tolerance=1e-10)[0] for c in contexts]
    held = free()
    T.release_idle_memory()
    idle = free() - held
    # blocks of 4 n bytes and more, of which the driver's pages of 2 MiB take up to a third more
    assert (1 << 30) < idle <= (4 << 30) * 4 // 3
    assert all(np.array_equal(v, x[0]) for v in x)
    assert np.array_equal(T.conjugate_gradient(contexts[0], csr, b, preconditioner_csr=csr, tolerance=1e-10)[0], x[0])
    for c in contexts:
        c.close()
    held = free()
    T.release_idle_memory()
    assert 0 <= free() - held <= (1 << 30) * 4 // 3


def test_sweep_values_that_do_not_fit(T):
    """The FP64 CG's sweep values take 400 bytes a row: with room for the exact triangular solves' memory alone, the
    solve takes those."""
    import scipy.sparse as sp
    import torch
    n = 1200000
    offs = [40000]   # few dependency levels
    U = sp.diags([np.full(n, 8.0)] + [np.full(n - o, -1.0) for o in offs], [0] + offs, shape=(n, n)).tocsr()
    csr = (U.indptr.astype(np.int64), U.indices.astype(np.int64), U.data)
    A, b = U + sp.triu(U, 1).T, np.random.default_rng(0).standard_normal(n)

    def solve(ctx):
        x = T.conjugate_gradient(ctx, csr, b, preconditioner_csr=csr, tolerance=1e-10)[0]
        assert np.linalg.norm(b - A @ x) <= 1.01e-10 * np.linalg.norm(b)

    T.release_idle_memory()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    ctx = T.Context()
    T.L.check(ctx._lib.nlgpu_set_option(ctx.handle, T.L.OPTION_GLOBAL_SWEEPS, 1))
    solve(ctx)   # its blocks are below 256 MiB and stay with the context
    need = before - torch.cuda.mem_get_info()[0]
    ctx.close()
    T.release_idle_memory()
    assert need < 1 << 30
    room = need + (160 << 20)   # the sweep values are 480 MB, more than what only the exact solves need
    filler = torch.empty(torch.cuda.mem_get_info()[0] - room, dtype=torch.uint8, device="cuda")
    try:
        ctx = T.Context()
        solve(ctx)
        ctx.close()
    finally:
        del filler
        torch.cuda.empty_cache()
        T.release_idle_memory()


def problem(T, n, stream=None, field=False, **model):
    from nonlocal_gb300.meshgen import structured_quad_mesh
    mesh = structured_quad_mesh(n, n - 3, "bilinear")
    pb = T.Problem2D.from_mesh(mesh, stream=stream)
    pb.set_model(T.Model2D(**dict(dict(influence="fast_polynomial", radius=(0.08, 0.08), local_weight=0.5), **model)))
    if field:
        pb.set_conductivity_field(np.random.default_rng(1).uniform(0.5, 2.0, mesh.n_elements * 4))
    pb.add_boundary(T.Boundary(edges=mesh.boundaries["left"], kind="temperature", value=1.0))
    pb.add_boundary(T.Boundary(edges=mesh.boundaries["right"], kind="flux", value=0.7))
    pb.find_neighbours()
    return pb


def close(a, b):
    # residuals of 1e-11 |b| and condition numbers below 1e4
    return np.linalg.norm(a - b) <= 2e-7 * np.linalg.norm(b)


@pytest.mark.parametrize("options", [{}, dict(precision="mixed"), dict(precision="mixed", coarse_aggregates=64)])
def test_callers_stream(T, options):
    import torch
    s = torch.cuda.Stream()
    ref = problem(T, 40).stationary(tolerance=1e-11, **options)[0]
    for _ in range(4):
        with torch.cuda.stream(s):   # work before the call, on memory that the allocators may exchange
            torch.randn(1 << 22, device="cuda")
        assert close(problem(T, 40, s.cuda_stream).stationary(tolerance=1e-11, **options)[0], ref)


def test_batches_in_turn(T):
    """Batches made and destroyed while their instances live on and are assembled again."""
    solvers = [T.NonstationaryHeatEquationSolver2D(problem(T, n), 1e-3) for n in (20, 31, 44)]
    ref = {}
    for k in range(6):
        for s in solvers:
            s.compute(np.zeros(s.problem.n_nodes))
        batch = T.BatchNonstationary(solvers)
        batch.set_method("mixed_illt" if k % 2 else "identity_fp64")
        for _ in range(3):
            batch.step(1.0, tolerance=1e-12)
        t = np.concatenate([batch.temperature(i) for i in range(3)])
        assert close(t, ref.setdefault(0, t))
        if k % 3 == 0:
            batch.close()
    fields = [problem(T, 30, field=True) for _ in range(3)]
    for k in range(4):
        for p in fields:
            p.conductivity_matrix("FULL")
        x = np.concatenate(T.solve_assembled_batch(fields, tolerance=1e-11, precision="mixed" if k % 2 else "fp64")[0])
        assert close(x, ref.setdefault(1, x))


def test_threads_of_every_solver(T):
    jobs = [lambda: problem(T, 45).stationary(tolerance=1e-11, precision="mixed")[0],
            lambda: problem(T, 40).stationary(tolerance=1e-11, precision="mixed", coarse_aggregates=100)[0],
            lambda: problem(T, 33, influence="exponential").stationary(tolerance=1e-11)[0],
            lambda: problem(T, 30, field=True).stationary(tolerance=1e-11, precision="mixed")[0],
            lambda: problem(T, 60, radius=(0.05, 0.05)).stationary(tolerance=1e-11, preconditioner="identity")[0],
            lambda: T.stationary_heat_equation_solver_1d(None, 500, 2, 1.0, 0.05, 0.5)]
    ref = [job() for job in jobs]
    bad = []

    def work(seed):
        for i in range(12):
            k = (5 * i + seed) % len(jobs)
            try:
                if not close(jobs[k](), ref[k]):
                    bad.append(k)
            except Exception as e:   # reported by the main thread
                bad.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(s,)) for s in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
