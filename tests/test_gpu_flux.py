"""The nodal flux in fixed point: scale invariance over the whole exponent range, non-finite temperatures, and the
rounding of the FP64 kernel."""
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


@pytest.mark.parametrize("element, nx, ny, influence, radius, p, q", [
    ("bilinear", 5, 3, "fast_polynomial", 0.5, 2, 1.0),
    ("bilinear", 40, 30, "fast_polynomial", 0.9, 2, 1.0),      # thousands of terms a lane
    ("bilinear", 100, 100, "fast_polynomial", 0.7, 2, 1.0),    # (30 000 an element: float-float lost 2e-14 of them)
    ("serendipity", 12, 10, "polynomial", 0.6, 2, 1.0),
    ("serendipity", 12, 10, "polynomial", 0.6, 8, 3.0),
    ("bilinear", 20, 15, "polynomial", 0.4, 2, 16.0),          # the steepest covered
    ("serendipity", 16, 12, "exponential", 0.4, 2, 0.5),
    ("serendipity", 16, 12, "exponential", 0.2, 2, 0.333),     # the ends of the covered range,
    ("serendipity", 16, 12, "exponential", 0.2, 2, 16.0),
    ("serendipity", 16, 12, "exponential", 0.2, 2, 17.0),      # outside,
    ("bilinear", 16, 12, "exponential", 0.005, 40, 2.0),       # d^(p / n) beyond single precision
    ("bilinear", 16, 12, "exponential", 1e-7, 2, 0.5),         # coordinates of millions of radii
])
@pytest.mark.parametrize("waves", [False, True])
def test_flux_rounds_as_the_fp64_kernel(element, nx, ny, influence, radius, p, q, waves):
    """Against the option's FP64 kernel: each of the two rounds the squared distance, the value, the weight and the sums
    to an eps or two; the waves cancel in the sums."""
    from nonlocal_gb300 import _lib
    from nonlocal_gb300 import thermal as T
    from nonlocal_gb300.meshgen import structured_quad_mesh
    if _lib.device_count() == 0:
        pytest.skip("no CUDA device")
    mesh = structured_quad_mesh(nx, ny, element, jitter=0.15, seed=2)
    x, y = mesh.nodes.T
    t = np.sin(31.0 * x) * np.cos(29.0 * y) if waves else 3.0 * x + y * y
    flux = []
    for kind in ("auto", "fp64"):
        pb = T.Problem2D.from_mesh(mesh)
        pb.set_model(T.Model2D(influence=influence, radius=(radius, radius), local_weight=0.0, p=p, q=q))
        pb.set_assembly_precision(kind)
        flux.append(np.array(pb.calc_flux(t)))
    assert np.isfinite(flux[1]).all()
    # what a relative change of d does to the value: q (p / n) d^(p / n) e^(-q d^(p / n)) <= p / n / e for the
    # exponential, p q / n at most for the polynomials
    eps = np.finfo(float).eps
    steep = p * q / 2.0 if influence != "exponential" else p / 2.0
    grad = 45.0 if waves else 4.0   # the largest |grad t|, and the quadrature's part of it
    # the normalisation makes the influence's integral 1 over the plane, at most 1 over the mesh; radii far below
    # an element's size see one point, whose share is bounded by the flux itself
    size = max(np.abs(flux[1]).max(), 1.1 * grad)
    assert np.abs(flux[0] - flux[1]).max() <= (4.0 * steep + 8.0) * eps * size
