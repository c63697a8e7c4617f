"""The 1D nonstationary solver on the GPU against the reference's own runs of
nonstationary_heat_equation_solver_1d (tests/golden/d1_nonstationary_*: the
temperature after every calc_step): quadratic elements with a bell kernel,
left temperature / right flux and a sin(pi x) source from zero; linear
elements with a triangle kernel, left flux / right temperature and a sin(pi x)
initial temperature; quadratic elements with a convection at both ends
(convection_1d: heat transfer and ambient temperature).  History within 1e-10
relative L2 per step."""
import numpy as np
import pytest

import golden_cases as gc

pytestmark = pytest.mark.gpu

SOLUTION_RTOL = 1e-10


@pytest.fixture(scope="module")
def lib():
    from nonlocal_gb300 import _lib, build
    build.build()
    _lib.load()
    if _lib.device_count() == 0:
        pytest.fail("no CUDA device visible to the nlgpu library")
    return _lib


def end(spec):
    kind = {"t": "temperature", "f": "flux", "c": "convection"}[spec[0]]
    if kind == "convection":   # c:<heat transfer>,<ambient temperature>
        h, t = spec[2:].split(",")
        return kind, (float(h), float(t))
    return kind, float(spec[2:])


@pytest.mark.parametrize("name", ["d1_nonstationary_quadratic", "d1_nonstationary_linear",
                                  "d1_nonstationary_convection"])
def test_nonstationary_1d_history(lib, name):
    from nonlocal_gb300 import thermal as T
    fx = gc.load(name)
    cfg = fx["config"]
    s = T.NonstationaryHeatEquationSolver1D(elements=int(cfg["elements"]), order=int(cfg["order"]), length=1.0,
                                            radius=float(cfg["radius"]), local_weight=float(cfg["local_weight"]),
                                            influence=cfg["influence"], conductivity=float(cfg["conductivity"]),
                                            capacity=float(cfg["capacity"]), density=float(cfg["density"]),
                                            time_step=float(cfg["dt"]))
    x = np.linspace(0.0, 1.0, s.n)
    initial = np.sin(np.pi * x) if cfg["initial"] == "sin" else None
    s.compute(left=end(cfg["left"]), right=end(cfg["right"]), initial=initial)
    if initial is not None:
        assert np.array_equal(s.temperature, initial)
    history = fx["history"]
    for k in range(history.shape[0]):
        t = s.calc_step(sin_source=cfg["source"] == "sin")
        err = np.linalg.norm(t - history[k]) / np.linalg.norm(history[k])
        assert err < SOLUTION_RTOL, (k, err)
    assert np.array_equal(s.temperature, t)


def test_nonstationary_1d_rejects_other_ends(lib):
    from nonlocal_gb300 import _lib as L
    from nonlocal_gb300 import thermal as T
    s = T.NonstationaryHeatEquationSolver1D(elements=10, order=1)
    with pytest.raises(L.NlgpuError):   # radiation ends are not built
        L.check(s.ctx._lib.nlgpu_nonstationary_1d_compute(s.ctx.handle, *s.args, L.BC_RADIATION, L.BC_FLUX, None,
                                                          None))
    with pytest.raises(L.NlgpuError):   # no compute yet
        s.calc_step(0.0, 0.0)


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("elements, radius, p1", [(1, 0.1, 1.0), (7, 0.3, 0.5), (15, 0.1, 1.0), (16, 0.2, 0.5), (33, 0.06, 0.4),
                                                  (120, 0.9, 0.5), (500, 0.3, 0.5)])
def test_band_factor_sizes(elements, radius, p1, order):
    """The blocked band factorisation where its blocks and bands meet edges: fewer rows than a block, a band
    narrower than a block, wider than the whole matrix and wider than the substitutions' prefetch, the last
    block partial; the stationary solve and the first implicit Euler step (temperature left, flux right) of the
    matrices restated densely."""
    from nonlocal_gb300 import thermal as T
    g, w = ((np.array([-1.0, 1.0]) / np.sqrt(3.0), np.ones(2)) if order == 1 else
            (np.array([-1.0, 0.0, 1.0]) * np.sqrt(0.6), np.array([5.0, 8.0, 5.0]) / 9.0))
    if order == 1:
        N, D = np.array([(1 - g) / 2, (1 + g) / 2]), np.array([-0.5 + 0 * g, 0.5 + 0 * g])
    else:
        N, D = np.array([g * (g - 1) / 2, 1 - g * g, g * (g + 1) / 2]), np.array([g - 0.5, -2 * g, g + 0.5])
    E, n, h = elements, elements * order + 1, 1.0 / elements
    x = (np.arange(E)[:, None] + (g + 1) / 2) * h
    K, C = np.zeros((n, n)), np.zeros((n, n))
    reach = int(np.floor(radius / h + 0.5)) if p1 < 0.999 else 0
    for e in range(E):
        ie = e * order + np.arange(order + 1)
        K[np.ix_(ie, ie)] += p1 * np.einsum("iq,jq,q->ij", D, D, w) / (h / 2)
        C[np.ix_(ie, ie)] += np.einsum("iq,jq,q->ij", N, N, w) * (h / 2)
        for f in range(max(0, e - reach), min(E, e + reach + 1)) if p1 < 0.999 else ():
            d = np.abs(x[e][:, None] - x[f][None, :])
            phi = np.where(d < radius, 0.75 / radius * (1 - (d / radius) ** 2), 0.0)
            K[np.ix_(ie, f * order + np.arange(order + 1))] += (1 - p1) * (D * w) @ phi @ (D * w).T
    b = np.zeros(n)
    for e in range(E):
        b[e * order:e * order + order + 1] += (N * w) @ np.sin(np.pi * x[e]) * (h / 2)
    b[-1] += 0.7
    t = T.stationary_heat_equation_solver_1d(elements=E, order=order, radius=radius, local_weight=p1, t_left=0.3,
                                             q_right=0.7)
    A, rhs = K[1:, 1:], b[1:] - K[1:, 0] * 0.3
    # both are backward stable: the residual of the solution, in units of its terms
    bound = 64 * n * np.finfo(float).eps * (np.abs(A) @ np.abs(t[1:]) + np.abs(rhs))
    assert t[0] == 0.3 and np.all(np.abs(A @ t[1:] - rhs) <= bound.max())
    s = T.NonstationaryHeatEquationSolver1D(elements=E, order=order, radius=radius, local_weight=p1, time_step=1e-3)
    s.compute(("temperature", 0.3), ("flux", 0.7), np.full(n, 0.5))
    u = s.calc_step()
    A = (C + 1e-3 * K)[1:, 1:]
    rhs = C[1:, 1:] @ np.full(n - 1, 0.5) - 1e-3 * K[1:, 0] * 0.3
    rhs[-1] += 1e-3 * 0.7
    bound = 64 * n * np.finfo(float).eps * (np.abs(A) @ np.abs(u[1:]) + np.abs(rhs))
    assert u[0] == 0.3 and np.all(np.abs(A @ u[1:] - rhs) <= bound.max())


@pytest.mark.parametrize("k", [0, 1019, 1021, 1022, 1023, -1018, -1021, -1022])
def test_pivots_at_the_ends_of_the_range(lib, k):
    """One local linear element of conductivity 2^k: its pivot's reciprocal is normal, subnormal, or the pivot the
    smallest normal number."""
    from nonlocal_gb300 import thermal as T
    t = T.stationary_heat_equation_solver_1d(None, 1, 1, 1.0, 0.1, 1.0, conductivity=2.0 ** k, t_left=1.0,
                                             q_right=2.0 ** (k - 1) if k > -1022 else 2.0 ** k, sin_source=False)
    assert np.array_equal(t, [1.0, 1.5 if k > -1022 else 2.0])


@pytest.mark.parametrize("elements, radius, p1, order", [(1, 0.1, 1.0, 1), (33, 0.06, 0.4, 2), (120, 0.9, 0.5, 1),
                                                         (500, 0.3, 0.5, 2)])
def test_cluster_of_eight(lib, monkeypatch, elements, radius, p1, order):
    """The factorisation's form for devices without room for a cluster of 16."""
    from nonlocal_gb300 import thermal as T

    class Eight(T.Context):
        def __init__(self, *args):
            super().__init__(*args)
            lib.check(self._lib.nlgpu_set_option(self.handle, lib.OPTION_BAND_CTAS, 8))

    monkeypatch.setattr(T, "Context", Eight)
    test_band_factor_sizes(elements, radius, p1, order)
    c = Eight()
    assert c._lib.nlgpu_set_option(c.handle, lib.OPTION_BAND_CTAS, 4) == 1
