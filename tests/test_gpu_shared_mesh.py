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
