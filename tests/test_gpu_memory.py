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
