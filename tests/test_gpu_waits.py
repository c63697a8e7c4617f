"""A wait between the CTAs of the one-launch FP32 ILLT application that runs out is reported by every call that
uses it.  NLGPU_OPTION_WAIT_LIMIT 0 lets each wait end at its first look that finds nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TIMEOUT = 8


@pytest.fixture(scope="module")
def T():
    from nonlocal_gb300 import _lib
    from nonlocal_gb300 import thermal
    if _lib.device_count() == 0:
        pytest.skip("no CUDA device")
    return thermal


def limit(T, pb, microseconds):
    T.L.check(pb._lib.nlgpu_set_option(pb.handle, T.L.OPTION_WAIT_LIMIT, microseconds))


def problem(T, field=False):
    from nonlocal_gb300.meshgen import structured_quad_mesh
    mesh = structured_quad_mesh(60, 50, "bilinear")
    pb = T.Problem2D.from_mesh(mesh)
    pb.set_model(T.Model2D(influence="fast_polynomial", radius=(0.08, 0.08), local_weight=0.5))
    if field:
        pb.set_conductivity_field(np.random.default_rng(1).uniform(0.5, 2.0, mesh.n_elements * 4))
    pb.add_boundary(T.Boundary(edges=mesh.boundaries["left"], kind="temperature", value=1.0))
    pb.add_boundary(T.Boundary(edges=mesh.boundaries["right"], kind="flux", value=0.7))
    pb.find_neighbours()
    return pb


def expect_timeout(T, call):
    with pytest.raises(T.L.NlgpuError) as e:
        call()
    assert e.value.status == TIMEOUT


def test_stationary(T):
    pb = problem(T)
    limit(T, pb, 0)
    expect_timeout(T, lambda: pb.stationary(precision="mixed", max_iterations=200))
    limit(T, pb, 2000000)
    assert pb.stationary(precision="mixed")[1].residual <= 1e-10


def test_batched_bicgstab(T):
    pbs = [problem(T, True) for _ in range(2)]
    for pb in pbs:
        pb.conductivity_matrix("FULL")
    limit(T, pbs[1], 0)
    expect_timeout(T, lambda: T.solve_assembled_batch(pbs, precision="mixed", max_iterations=50))
    limit(T, pbs[1], 2000000)
    assert all(r.residual <= 1e-10 for r in T.solve_assembled_batch(pbs, precision="mixed")[1])


def test_batched_steps(T):
    solvers = []
    for _ in range(2):
        s = T.NonstationaryHeatEquationSolver2D(problem(T), 1e-3)
        s.compute(np.zeros(s.problem.n_nodes))
        solvers.append(s)
    limit(T, solvers[0].problem, 0)
    batch = T.BatchNonstationary(solvers)
    batch.set_method("mixed_illt")
    expect_timeout(T, lambda: batch.step(1.0, tolerance=1e-10, max_iterations=500))


def test_learned(T):
    pb = problem(T)
    pb.conductivity_matrix("FULL")
    pb.train_learned_preconditioner(right_hand_sides=2, epochs=1)
    x = np.random.default_rng(0).standard_normal(pb.n_nodes).astype(np.float32)
    pb.learned_loss_grad(x, x)
    limit(T, pb, 0)
    expect_timeout(T, lambda: pb.learned_loss_grad(x, x))
    expect_timeout(T, lambda: pb.train_learned_preconditioner(right_hand_sides=2, epochs=1))
    limit(T, pb, 2000000)
    pb.learned_loss_grad(x, x)


def test_option_values(T):
    pb = problem(T)
    assert pb._lib.nlgpu_set_option(pb.handle, T.L.OPTION_WAIT_LIMIT, -1) == 1
