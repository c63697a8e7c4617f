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


def exact_inner(mesh, pb, model):
    """The inner matrix by pairs of elements in extended precision (p = n = 2, without the influence's normalisation), and
    beside it the sums of its terms' magnitudes."""
    L = np.longdouble
    qc, jac, der = (v.astype(L) for v in pb.quadrature())
    w = pb.basis()["basis_weights"].astype(L)
    off, lst = pb.neighbours()
    lam = np.array(model.conductivity * (2 if len(model.conductivity) == 1 else 1), dtype=L)
    K, M = (np.zeros((mesh.n_nodes, mesh.n_nodes), dtype=L) for _ in range(2))
    q = 1.0 if model.influence == "fast_polynomial" else model.q
    for e in range(mesh.n_elements):
        for f in lst[off[e]:off[e + 1]]:
            d = (((qc[e][:, None] - qc[f][None]) / np.array(model.radius, dtype=L)) ** 2).sum(-1)
            phi = np.exp(-L(q) * d) if model.influence == "exponential" else np.where(d < 1, 1 - d, 0) ** int(q)
            phi = phi * w[:, None] * w[None]
            g = der[f] * lam
            at = np.ix_(mesh.elements[e], mesh.elements[f])
            K[at] += sum(der[e][:, :, k] @ phi @ g[:, :, k].T for k in (0, 1))
            M[at] += sum(abs(der[e][:, :, k]) @ phi @ abs(g[:, :, k]).T for k in (0, 1))
    return K, M


def errors(T, mesh, model, fixed):
    """Per assembly precision: the largest error of an entry against its terms' sum, the largest against the root of its
    diagonal entries' product, and the root mean square of the latter."""
    pb = T.Problem2D.from_mesh(mesh)
    pb.set_model(model)
    pb.add_boundary(T.Boundary(edges=fixed, kind="temperature", value=1.0))
    pb.find_neighbours()
    K, M = exact_inner(mesh, pb, model)
    diag = np.sqrt(np.abs(K.diagonal()))
    out = {}
    for kind in ("ff", "auto", "fp64"):
        pb.set_assembly_precision(kind)
        pb.conductivity_matrix("FULL")
        rp, col, val = pb.matrix("inner")
        row = np.repeat(np.arange(mesh.n_nodes), np.diff(rp))
        free = ~np.isin(row, fixed) & ~np.isin(col, fixed)
        row, col, val = row[free], col[free], val[free]
        ref, mag = K[row, col], M[row, col]
        err = np.abs(val / ((val * ref).sum() / (ref * ref).sum()) - ref)   # up to the influence's normalisation
        scaled = err / (diag[row] * diag[col])
        out[kind] = (float((err / np.where(mag > 0, mag, 1)).max()), float(scaled.max()), float(np.sqrt((scaled ** 2).mean())))
    return out


@pytest.mark.parametrize("aspect, conductivity", [
    ("x", (1e6, 1.0)),        # stretched elements, the conductivity makes up for it: a common power of two
    ("x", (1.0,)),
    ("x", (1.0, 0.0)),        # nothing in one direction
    ("both", (1.0,)),         # elements stretched one way beside ones stretched the other: FP64 for FP64 solves
])
def test_stretched_elements(T, aspect, conductivity):
    """As accurate as the FP64 kernel, whose entries are sums of at most 81 pairs of 16 products: 8 eps of the diagonal
    (of the terms where the entries' scales differ by powers of the stretch)."""
    from nonlocal_gb300.meshgen import BILINEAR, QuadMesh
    rng = np.random.default_rng(5)
    if aspect == "x":
        xs, ys, radius, move = np.arange(7) * 1000.0, np.arange(6) * 1.0, (2100.0, 2.1), (200.0, 0.2)
    else:
        xs = np.concatenate([[0.0], np.cumsum([1000.0] * 3 + [1.0] * 3)])
        ys = np.concatenate([[0.0], np.cumsum([1.0, 1.0, 30.0, 1000.0, 1000.0])])
        radius, move = (2100.0, 2100.0), (0.2, 0.2)
    X, Y = np.meshgrid(xs, ys)
    nodes = np.stack([X.ravel(), Y.ravel()], 1) + rng.uniform(-1.0, 1.0, (42, 2)) * np.array(move)
    el = np.array([[j * 7 + i, j * 7 + i + 1, (j + 1) * 7 + i + 1, (j + 1) * 7 + i] for j in range(5) for i in range(6)])
    model = T.Model2D(influence="fast_polynomial", radius=radius, local_weight=0.0, conductivity=conductivity)
    e = errors(T, QuadMesh(BILINEAR, nodes, el.astype(np.int64), {}), model, np.array([[0, 7]]))
    which = 1 if aspect == "x" else 0
    eps = np.finfo(float).eps
    assert e["fp64"][which] <= 8 * eps
    assert e["auto"][which] <= 8 * eps
    assert e["ff"][which] <= 1e-12


@pytest.mark.parametrize("influence, q", [("fast_polynomial", 1.0), ("polynomial", 1.0), ("polynomial", 3.0),
                                          ("polynomial", 16.0)])
@pytest.mark.parametrize("element, nx, ny, radius", [("bilinear", 14, 12, 0.25), ("serendipity", 8, 6, 0.35)])
def test_entries_at_the_edge_of_the_influence(T, influence, q, element, nx, ny, radius):
    """Entries that only pairs at the horizon make, however small, keep their digits: a pair's values are good to 2^-52
    of its largest one, of which an entry's own terms are 2^-17 or more in a block of 64 on a jittered mesh."""
    from nonlocal_gb300.meshgen import structured_quad_mesh
    mesh = structured_quad_mesh(nx, ny, element, jitter=0.2, seed=1)
    model = T.Model2D(influence=influence, radius=(radius, radius), local_weight=0.0, q=q, conductivity=(2.0, 1.0))
    e = errors(T, mesh, model, mesh.boundaries["left"])
    assert e["auto"][0] <= 2.0 ** -35
    assert e["ff"][0] <= 2.0 ** -35
    # against the diagonal: the FP64 kernel's bound as for the stretched elements, q times for the power
    assert e["auto"][1] <= 32 * q ** 0.5 * np.finfo(float).eps


@pytest.mark.parametrize("q", [0.333, 0.5, 2.0, 8.0, 16.0])
@pytest.mark.parametrize("element, nx, ny, radius", [("bilinear", 14, 12, 0.25), ("serendipity", 8, 6, 0.35)])
def test_exponentials_are_as_accurate_as_fp64(T, q, element, nx, ny, radius):
    """FP64 solves: over thousands of entries the root mean square error is that of the FP64 kernel or less; 10 % for the
    sample."""
    from nonlocal_gb300.meshgen import structured_quad_mesh
    mesh = structured_quad_mesh(nx, ny, element, jitter=0.2, seed=1)
    model = T.Model2D(influence="exponential", radius=(radius, radius), local_weight=0.0, q=q, conductivity=(2.0, 1.0))
    e = errors(T, mesh, model, mesh.boundaries["left"])
    assert e["auto"][2] <= 1.1 * e["fp64"][2]


def test_coordinates_of_a_billion_radii(T):
    """Fixed-point coordinates have a unit of 2^-58 of the largest: far from the origin the FP64 kernel takes over."""
    from nonlocal_gb300.meshgen import structured_quad_mesh
    mesh = structured_quad_mesh(6, 5, "bilinear", width=6.0, height=5.0)
    mesh.nodes += 2.0 ** 31
    model = T.Model2D(influence="fast_polynomial", radius=(2.25, 2.25), local_weight=0.3)
    _, (ff, auto, fp) = matrices(T, mesh, model)
    scale = np.abs(fp[0]).max()
    for a, x, b in zip(ff, auto, fp):
        assert np.abs(x - b).max(initial=0.0) <= 32 * 2.0 ** -53 * 20 * scale
        assert np.abs(a - b).max(initial=0.0) <= 32 * 2.0 ** -53 * 20 * scale
