"""The full rows filled from the upper storage: solves whose residual is formed on the host from the upper matrix,
for each way of filling (short rows by search, one to 32 rows a warp, scattered numbering, non-symmetric rows, the
map kept with radiation)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("element, nx, ny, radius, kind", [
    ("bilinear", 23, 17, None, "plain"),              # a classical problem: 9 entries a row
    ("serendipity", 9, 7, 0.35, "plain"),
    ("serendipity", 9, 7, 0.35, "scattered"),
    ("bilinear", 45, 41, 0.8, "plain"),               # beyond 1024 entries a row: one row a warp,
    ("bilinear", 45, 41, 0.8, "scattered"),
    ("bilinear", 110, 100, 0.21, "plain"),            # two,
    ("bilinear", 171, 173, 0.12, "plain"),            # and six, a partial last block
    ("bilinear", 45, 41, 0.8, "field"),
    ("bilinear", 21, 18, 0.3, "field"),
    ("serendipity", 8, 6, 0.4, "radiation"),
])
def test_residual_from_the_upper_storage(element, nx, ny, radius, kind):
    import scipy.sparse as sp
    from nonlocal_gb300 import _lib
    from nonlocal_gb300 import thermal as T
    from nonlocal_gb300.meshgen import relabel_nodes, structured_quad_mesh
    if _lib.device_count() == 0:
        pytest.skip("no CUDA device")
    mesh = structured_quad_mesh(nx, ny, element, jitter=0.2, seed=4)
    if kind == "scattered":
        mesh = relabel_nodes(mesh, np.random.default_rng(0).permutation(mesh.n_nodes))
    pb = T.Problem2D.from_mesh(mesh)
    pb.set_model(T.Model2D(influence="polynomial", radius=(radius or 0.1,) * 2, local_weight=1.0 if radius is None else 0.5))
    if kind == "field":
        pb.set_conductivity_field(np.random.default_rng(1).uniform(0.5, 2.0, mesh.n_elements * 4))
    left = mesh.boundaries["left"][:-2] if kind == "radiation" else mesh.boundaries["left"]   # apart from "up"
    pb.add_boundary(T.Boundary(edges=left, kind="temperature", value=1.0))
    pb.add_boundary(T.Boundary(edges=mesh.boundaries["right"], kind="flux", value=0.7))
    if kind == "radiation":   # at vanishing emissivity: the map's path, a linear problem
        pb.add_boundary(T.Boundary(edges=mesh.boundaries["up"], kind="radiation", emissivity=1e-300))
    if radius is not None:
        pb.find_neighbours()
    pb.conductivity_matrix("FULL")
    x = T.solve_assembled_batch([pb], tolerance=1e-12, max_iterations=5000)[0][0]
    rp, col, val = pb.matrix("inner")
    A = sp.csr_matrix((val, col, rp), shape=(mesh.n_nodes,) * 2)
    if kind != "field":
        A = A + sp.triu(A, 1).T
    b = pb.rhs()[0]
    assert np.linalg.norm(b - A @ x) <= 2e-12 * np.linalg.norm(b)
