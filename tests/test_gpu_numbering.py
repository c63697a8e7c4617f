"""Meshes whose nodes are numbered at random (as a mesher may number them) or after cuthill_mckee."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from nonlocal_gb300 import _lib
    if _lib.device_count() == 0:
        pytest.skip("no CUDA device")
    return _lib


def problem(mesh, radius, influence="polynomial"):
    from nonlocal_gb300 import thermal as T
    pb = T.Problem2D.from_mesh(mesh)
    pb.set_model(T.Model2D(influence=influence, radius=(radius, radius), local_weight=0.5))
    pb.add_boundary(T.Boundary(edges=mesh.boundaries["left"], kind="temperature", value=1.0))
    pb.find_neighbours()
    return pb


def test_one_kernel_fills_the_full_rows(lib):
    """Long rows of scattered columns take the kernel that short rows take: the same launches."""
    from nonlocal_gb300.meshgen import relabel_nodes, structured_quad_mesh
    mesh = structured_quad_mesh(45, 41, "bilinear")
    mesh = relabel_nodes(mesh, np.random.default_rng(0).permutation(mesh.n_nodes))
    launches = []
    for radius in (0.1, 0.8):   # about 60 entries a row, and beyond 1024
        pb = problem(mesh, radius)
        before = lib.kernel_launches()
        pb.conductivity_matrix("FULL")
        launches.append(lib.kernel_launches() - before)
    assert launches[0] == launches[1]


@pytest.mark.parametrize("element, nx, ny, radius", [("bilinear", 60, 50, 0.1), ("bilinear", 60, 50, 0.03),
                                                     ("serendipity", 30, 20, 0.12)])
def test_pattern_of_scattered_nodes(lib, element, nx, ny, radius):
    """Words of a few bits and of many in one row: the pattern of randomly numbered nodes, and of nodes of which a
    half keeps its order, is the permuted pattern of the mesh as numbered row by row."""
    from nonlocal_gb300.meshgen import relabel_nodes, structured_quad_mesh
    mesh = structured_quad_mesh(nx, ny, element)
    n = mesh.n_nodes

    def pairs(m, to_row):
        pb = problem(m, radius)
        pb.conductivity_matrix("FULL")
        out = []
        for which in ("inner", "bound"):
            rp, col, _ = pb.matrix(which)
            row = np.repeat(np.arange(n), np.diff(rp))
            assert all(np.all(np.diff(col[rp[r]:rp[r + 1]]) > 0) for r in range(n))
            a, b = to_row[row], to_row[col]
            out.append(np.unique(np.minimum(a, b) * n + np.maximum(a, b) if which == "inner" else a * n + b))
        return out

    expected = pairs(mesh, np.arange(n))
    rng = np.random.default_rng(3)
    half = np.arange(n)
    half[n // 2:] = n // 2 + rng.permutation(n - n // 2)
    for perm in (rng.permutation(n), half):
        for e, g in zip(expected, pairs(relabel_nodes(mesh, perm), np.argsort(perm))):
            assert np.array_equal(e, g)


@pytest.mark.parametrize("step, one_launch", [(100, True), (5000, False)])
def test_sweeps_by_the_reach_of_the_columns(lib, step, one_launch):
    """160 000 rows of five entries, 0.8 million in a triangle: columns within a CTA's rows or the next take the
    one-launch application, columns tens of CTAs away a launch per sweep; both give M^-1 x."""
    import scipy.sparse as sp
    from nonlocal_gb300 import thermal as T
    n, k = 160000, 5
    offs = [step * j for j in range(1, k + 1)]
    U = sp.diags([np.full(n, 4.0 * k)] + [np.full(n - o, -1.0) for o in offs], [0] + offs, shape=(n, n)).tocsr()
    pre = T.EigenILLTPreconditioner()
    assert pre.compute((U.indptr, U.indices, U.data)).computation_info() == pre.SUCCESS
    x = np.random.default_rng(0).standard_normal(n).astype(np.float32)
    pre.solve_f32(x)
    before = lib.kernel_launches()
    y = pre.solve_f32(x, 6)
    launches = lib.kernel_launches() - before
    assert launches == 1 if one_launch else launches >= 12
    # a row's off-diagonal sum is at most 5 / 20 of its diagonal: six sweeps of each triangle leave 0.26^7 of the
    # vector or less, and FP32 a few 1e-7
    ref = pre.solve(x.astype(np.float64))
    assert np.linalg.norm(y - ref) <= 3e-4 * np.linalg.norm(ref)


@pytest.mark.parametrize("every, one_launch", [(0, True), (20, True), (5, False)])
def test_sweeps_by_the_share_of_far_columns(lib, every, one_launch):
    """160 000 rows of five near entries, and one 20 000 columns away on none of them, on every 20th (0.9 %
    of the entries) and on every 5th (3.4 %): a mean reach below four CTAs in all three; both forms give M^-1 x."""
    import scipy.sparse as sp
    from nonlocal_gb300 import thermal as T
    n, k, away = 160000, 5, 20000
    offs = [100 * j for j in range(1, k + 1)]
    U = sp.diags([np.full(n, 4.0 * (k + 1))] + [np.full(n - o, -1.0) for o in offs], [0] + offs, shape=(n, n))
    if every:
        rows = np.arange(0, n - away, every)
        U = U + sp.coo_matrix((np.full(rows.size, -1.0), (rows, rows + away)), shape=(n, n))
    U = U.tocsr()
    U.sort_indices()
    pre = T.EigenILLTPreconditioner()
    assert pre.compute((U.indptr, U.indices, U.data)).computation_info() == pre.SUCCESS
    x = np.random.default_rng(0).standard_normal(n).astype(np.float32)
    pre.solve_f32(x)
    before = lib.kernel_launches()
    y = pre.solve_f32(x, 6)
    launches = lib.kernel_launches() - before
    assert launches == 1 if one_launch else launches >= 12
    # a row's off-diagonal sum is at most 6 / 24 of its diagonal, as above
    ref = pre.solve(x.astype(np.float64))
    assert np.linalg.norm(y - ref) <= 3e-4 * np.linalg.norm(ref)


@pytest.mark.parametrize("n, k, one_launch", [(150000, 7, True), (190000, 7, False), (290000, 5, True)])
def test_sweeps_by_the_length_of_the_rows(lib, n, k, one_launch):
    """Near columns: 1.05 million entries of seven a row take the one-launch application, 1.33 million do not, and
    of five a row 1.45 million do; both forms give M^-1 x."""
    import scipy.sparse as sp
    from nonlocal_gb300 import thermal as T
    offs = [100 * j for j in range(1, k + 1)]
    U = sp.diags([np.full(n, 4.0 * k)] + [np.full(n - o, -1.0) for o in offs], [0] + offs, shape=(n, n)).tocsr()
    pre = T.EigenILLTPreconditioner()
    assert pre.compute((U.indptr, U.indices, U.data)).computation_info() == pre.SUCCESS
    x = np.random.default_rng(0).standard_normal(n).astype(np.float32)
    pre.solve_f32(x)
    before = lib.kernel_launches()
    y = pre.solve_f32(x, 6)
    launches = lib.kernel_launches() - before
    assert launches == 1 if one_launch else launches >= 12
    # a row's off-diagonal sum is at most a quarter of its diagonal, as above
    ref = pre.solve(x.astype(np.float64))
    assert np.linalg.norm(y - ref) <= 3e-4 * np.linalg.norm(ref)
