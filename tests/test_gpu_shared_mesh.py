"""Solvers on one mesh run on streams of their own: what the mesh holds for them (the connectivity built on first
use) is whole before a second solver takes it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(semgb, mesh, seed):
    rng = np.random.default_rng(seed)
    s = semgb.Solver(mesh, 2e-4)
    s.set_kernel(semgb.KERNEL_ELEMENT)
    s.set_sources(rng.choice(mesh.n_elem, 3), rng.standard_normal((3, 4)).astype(np.float32))
    return s


def test_element_solvers_started_at_once(semgb_lib, cuda_device):
    semgb = semgb_lib

    def run(waited):
        mesh = semgb.Mesh(40, 36, 38, 400.0, 360.0, 380.0, 4)
        solvers = [_solver(semgb, mesh, k) for k in range(3)]
        for s in solvers:
            s.step(4)
            if waited:
                s.synchronize()
        return [s.pressure() for s in solvers]

    for got, want in zip(run(False), run(True)):
        # (the element path's float atomics have no fixed order)
        assert np.abs(want).max() > 0 and np.abs(got - want).max() <= 1e-5 * np.abs(want).max()


@pytest.mark.parametrize("nodes", [False, True])
def test_model_changed_behind_steps_under_way(semgb_lib, cuda_device, nodes):
    """A model set right after a call of steps does not reach the steps of that call, whose mass is formed on
    the solver's stream behind earlier steps."""
    semgb = semgb_lib

    def run(waited):
        mesh = semgb.Mesh(48, 44, 46, 480.0, 440.0, 460.0, 4)
        rng = np.random.default_rng(5)

        def model(c):
            if nodes:
                mesh.set_slowness2(np.full(mesh.n_nodes, 1.0 / c ** 2, np.float32))
            else:
                mesh.set_velocity(np.full(mesh.n_elem, c, np.float32))

        model(2000.0)
        s = semgb.Solver(mesh, 2e-4)
        s.set_pressure(semgb.LEVEL_CURRENT, rng.standard_normal(mesh.n_nodes).astype(np.float32))
        for c in (2500.0, 1500.0, 3000.0):
            s.step(100)
            if waited:
                s.synchronize()
            model(c)
        return s.pressure()

    got, want = run(False), run(True)
    assert np.isfinite(want).all() and np.abs(want).max() > 0 and np.array_equal(got, want)
