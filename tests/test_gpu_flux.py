"""The float-float nodal flux: scale invariance over the whole exponent range, and non-finite temperatures."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("element", ["bilinear", "serendipity"])
@pytest.mark.parametrize("influence, p", [("fast_polynomial", 2), ("polynomial", 4), ("exponential", 2)])
def test_flux_scaling_and_non_finite_temperatures(element, influence, p):
    from nonlocal_gb300 import _lib
    from nonlocal_gb300 import thermal as T
    from nonlocal_gb300.meshgen import structured_quad_mesh
    if _lib.device_count() == 0:
        pytest.skip("no CUDA device")
    mesh = structured_quad_mesh(13, 7, element, jitter=0.2, seed=1, width=13.0, height=7.0)
    pb = T.Problem2D.from_mesh(mesh)
    pb.set_model(T.Model2D(influence=influence, radius=(2.1, 1.6), local_weight=0.4, p=p, conductivity=(2.0, 0.5)))
    t = np.random.default_rng(3).standard_normal(mesh.n_nodes)
    f0 = pb.calc_flux(t)
    # every operation before and after the sums is exact under a power of two
    for k in (600, -600, 0):
        for a, b in zip(pb.calc_flux(np.ldexp(t, k)), f0):
            assert np.array_equal(a, np.ldexp(b, k)), k
    assert all(np.array_equal(v, np.zeros_like(v)) for v in pb.calc_flux(np.full(mesh.n_nodes, 0.0)))
    # an infinite temperature: the FP64 kernel's sums; out of its reach the finite ones, to the rounding
    # of a sum of at most 13 * 7 * 9 terms
    u = t.copy()
    corner = int(np.argmin(mesh.nodes.sum(axis=1)))
    u[corner] = np.inf
    far = mesh.nodes[:, 0] > 8.0
    scale = max(np.abs(v).max() for v in f0)
    for a, b in zip(pb.calc_flux(u), f0):
        assert not np.isfinite(a[corner])
        assert np.abs(a[far] - b[far]).max() <= 819 * 4 * np.finfo(float).eps * scale
