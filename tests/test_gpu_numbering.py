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
