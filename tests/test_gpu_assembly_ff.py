"""The float-float and fixed-point pair assembly against the FP64 kernel: more candidates than one list holds, one element,
influence that ends inside the neighbourhood, and element and conductivity scales far from one."""
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


def matrices(T, mesh, model, field=None):
    pb = T.Problem2D.from_mesh(mesh)
    pb.set_model(model)
    if field is not None:
        pb.set_conductivity_field(field)
    pb.add_boundary(T.Boundary(edges=mesh.boundaries["left"], kind="temperature", value=1.0))
    pb.find_neighbours()
    out = []
    for kind in ("ff", "auto", "fp64"):
        pb.set_assembly_precision(kind)
        pb.conductivity_matrix("FULL")
        out.append([pb.matrix(which)[2].copy() for which in ("inner", "bound")])
    return pb, out


# a block's error is that of 48-bit influence values, 2^-46 of its terms' sum; the largest entry is at least a
# twentieth of that sum here, and the bar the project's 1e-12 of the largest entry
@pytest.mark.parametrize("element, nx, ny, size, radius, influence, p, conductivity", [
    ("bilinear", 1, 1, 1.0, 1.0, "exponential", 2, (1.0,)),
    ("serendipity", 1, 1, 1.0, 0.7, "polynomial", 2, (1.0,)),
    ("bilinear", 41, 40, 1.0, 0.55, "fast_polynomial", 2, (1.0, 0.2)),      # beyond 1024 neighbours
    ("serendipity", 9, 7, 1.0, 0.3, "fast_polynomial", 2, (2.0, 1.0, 0.5)),
    ("bilinear", 17, 3, 1e-6, 2e-7, "polynomial", 4, (1.0,)),
    ("serendipity", 6, 5, 1e5, 3e4, "exponential", 2, (1.0, 3.0)),
    ("bilinear", 7, 6, 1.0, 0.4, "exponential", 1, (1e-25,)),               # n = 1: not in fixed point
    ("bilinear", 9, 6, 1.0, 0.02, "exponential", 2, (1.0,)),                # values down to where they end
    ("serendipity", 5, 3, 1.0, 0.9, "polynomial", 6, (1.0, 7.0)),
    ("serendipity", 5, 4, 1.0, 0.4, "polynomial", 2, (1e28,)),
])
def test_float_float_against_fp64(T, element, nx, ny, size, radius, influence, p, conductivity):
    from nonlocal_gb300.meshgen import structured_quad_mesh
    mesh = structured_quad_mesh(nx, ny, element, jitter=0.2, seed=2, width=size, height=size)
    model = T.Model2D(influence=influence, radius=(radius, 0.8 * radius), local_weight=0.3, n=1 if p == 1 else 2, p=p,
                      conductivity=conductivity)
    for field in (None, np.linspace(0.5, 2.0, mesh.n_elements * (4 if element == "bilinear" else 9))):
        if field is not None and len(conductivity) > 1:
            continue
        pb, (ff, auto, fp) = matrices(T, mesh, model, field)
        assert pb.assembly_tuning()["warps"] in (16, 32)
        scale = np.abs(fp[0]).max()
        for a, x, b in zip(ff, auto, fp):
            assert np.abs(a - b).max(initial=0.0) <= 1e-12 * scale
            # FP64 solves: the FP64 kernel's own rounding, dots of 9 and 18 terms, 32 2^-53 of the terms' sum
            assert np.abs(x - b).max(initial=0.0) <= 32 * 2.0 ** -53 * 20 * scale


def test_non_finite_field_reaches_its_rows(T):
    from nonlocal_gb300.meshgen import structured_quad_mesh
    mesh = structured_quad_mesh(12, 4, "bilinear", width=12.0, height=4.0)
    field = np.ones(mesh.n_elements * 4)
    clean = matrices(T, mesh, T.Model2D(influence="fast_polynomial", radius=(1.5, 1.5), local_weight=0.3), field)[1][0][0]
    field[4 * 30] = np.nan
    pb, (ff, auto, fp) = matrices(T, mesh, T.Model2D(influence="fast_polynomial", radius=(1.5, 1.5), local_weight=0.3), field)
    rowptr = pb.matrix("inner")[0]
    for r in mesh.elements[30]:
        assert not np.isfinite(ff[0][rowptr[r]:rowptr[r + 1]]).all()
        assert not np.isfinite(auto[0][rowptr[r]:rowptr[r + 1]]).all()
    # beyond the influence of the element nothing changes, to the order of the sums
    far = np.isfinite(fp[0])
    assert far.any() and np.abs(ff[0] - clean)[far].max() <= 1e-14 * np.abs(clean).max()


def test_powers_beyond_single_precision(T):
    """Elements several radii wide and a steep exponential: d^(p / n) overflows a float, where the value is 0."""
    from nonlocal_gb300.meshgen import structured_quad_mesh
    mesh = structured_quad_mesh(16, 12, "bilinear", jitter=0.15, seed=2)
    model = T.Model2D(influence="exponential", radius=(0.005, 0.005), local_weight=0.3, p=40, q=2.0)
    _, (ff, _, fp) = matrices(T, mesh, model)
    scale = np.abs(fp[0]).max()
    assert np.isfinite(fp[0]).all()
    for a, b in zip(ff, fp):   # values of 48 bits whose exponent is good to p / n times that
        assert np.abs(a - b).max(initial=0.0) <= 1e-12 * scale
