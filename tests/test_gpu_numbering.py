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
