"""Runs of 16 steps are launched one by one until there were eight (branches of a group: four) since the last
change and replayed from a graph after that: calls on both sides of the switch, and a change of the sources that takes the graph
away, give the bits of single steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("calls", [[16] * 11, [128, 16, 17], [129, 144], [144, 1, 16], [100, 100]])
def test_launched_then_replayed(semgb_lib, cuda_device, calls):
    semgb = semgb_lib
    n = sum(calls)
    out = []
    for single in (False, True):
        mesh = semgb.Mesh(9, 8, 7, 90.0, 80.0, 70.0, 2)
        mesh.set_velocity(np.linspace(1500, 3000, mesh.n_elem).astype(np.float32))
        s = semgb.Solver(mesh, 2e-4)
        s.set_sponge(2, 0.1)
        s.set_receiver_nodes(np.arange(0, mesh.n_nodes, 37))
        got = []
        for elements in ([200, 201, 200], [130]):
            w = np.random.default_rng(len(elements)).standard_normal((len(elements), 2 * n)).astype(np.float32)
            s.set_sources(np.array(elements), w)
            for c in [1] * n if single else calls:
                s.step(c)
            got.append(s.pressure())
        out.append((got, s.traces()))
    for a, b in zip(out[0][0], out[1][0]):
        assert np.array_equal(a, b)
    assert np.array_equal(out[0][1], out[1][1]) and np.abs(out[0][1]).max() > 0


@pytest.mark.parametrize("calls", [[16] * 10 + [3], [145], [64, 17, 64]])
@pytest.mark.parametrize("kind", ["network", "batch", "branches"])
def test_launched_then_replayed_with_boundary_batch_and_group(semgb_lib, cuda_device, kind, calls):
    semgb = semgb_lib
    n = sum(calls)
    out = []
    for single in (False, True):
        meshes, solvers = [], []
        for k in range(1 if kind != "branches" else 3):
            mesh = semgb.Mesh(9 + k, 8, 7, 90.0 + 10 * k, 80.0, 70.0, 2 + k)
            mesh.set_velocity(np.linspace(1500, 3000, mesh.n_elem).astype(np.float32))
            w = np.random.default_rng(k).standard_normal((2, n)).astype(np.float32)
            s = semgb.Batch(mesh, 2e-4, 2) if kind == "batch" else semgb.Solver(mesh, 2e-4)
            s.set_sponge(2, 0.1)
            s.set_receiver_nodes(np.arange(0, mesh.n_nodes, 37))
            s.set_sources(np.array([200, 201]), w)
            meshes.append(mesh)
            solvers.append(s)
        stepped = solvers[0]
        if kind == "network":
            stepped = semgb.Abc(solvers[0], semgb.Mlp(3), 0)
        if kind == "branches":
            stepped = semgb.Group(solvers, semgb.GROUP_BRANCHES)
        for c in [1] * n if single else calls:
            stepped.step(c)
        out.append([x for s in solvers
                    for x in (s.traces(), *([s.pressure(0), s.pressure(1)] if kind == "batch" else [s.pressure()]))])
    assert all(np.array_equal(a, b) and np.abs(a).max() > 0 for a, b in zip(*out))
