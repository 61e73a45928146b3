"""Runs of 16 steps are launched one by one until there were eight since the last change and replayed from
a graph after that: calls on both sides of the switch, and a change of the sources that takes the graph
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
