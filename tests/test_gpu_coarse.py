"""The coarse correction at the sizes where AP's rows change form: a handful of aggregates, rows of few
aggregates (summed in fixed point), rows of more than 128 (kept as runs), Dirichlet columns inside the rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("element, n, radius, aggregates, fewer", [
    ("bilinear", 64, 0.16, 4, 1.0), ("bilinear", 64, 0.16, 100, 2.0), ("bilinear", 64, 0.16, 2048, 2.0),
    ("serendipity", 33, 0.2, 60, 1.5), ("serendipity", 33, 0.2, 700, 1.5), ("bilinear", 5, 0.5, 9, 1.0)])
def test_aggregates(element, n, radius, aggregates, fewer):
    from nonlocal_gb300 import _lib
    from nonlocal_gb300 import thermal as T
    from nonlocal_gb300.meshgen import structured_quad_mesh
    if _lib.device_count() == 0:
        pytest.skip("no CUDA device")
    mesh = structured_quad_mesh(n, n, element, jitter=0.2, seed=5)
    pb = T.Problem2D.from_mesh(mesh)
    pb.set_model(T.Model2D(influence="fast_polynomial", radius=(radius, radius), local_weight=0.5))
    pb.add_boundary(T.Boundary(edges=mesh.boundaries["left"], kind="temperature", value=1.0))
    pb.add_boundary(T.Boundary(edges=mesh.boundaries["right"], kind="flux", value=1.0))
    pb.find_neighbours()
    ref, _ = pb.stationary(tolerance=1e-13, max_iterations=20000)
    _, plain = pb.stationary(tolerance=1e-12, max_iterations=20000, precision="mixed")
    t, rep = pb.stationary(tolerance=1e-12, max_iterations=20000, precision="mixed", coarse_aggregates=aggregates)
    assert rep.residual <= 1e-12
    assert np.linalg.norm(t - ref) <= 1e-9 * np.linalg.norm(ref)
    assert rep.iterations * fewer <= plain.iterations + 2, (rep.iterations, plain.iterations)
