"""Order 1 looks up a CTA's sources and receivers before its march: no sources or receivers, one of each,
and more source nodes than a CTA has threads, on boxes of several tiles and chunks and a far edge;
a run gives the bits of its steps one by one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc,nrec", [(0, 3), (1, 0), (1, 1), (128, 129), (300, 2000)])
@pytest.mark.parametrize("box", [(32, 21, 33), (17, 64, 16)])
def test_run_equals_single_steps(semgb_lib, cuda_device, box, nsrc, nrec):
    semgb = semgb_lib
    ex, ey, ez = box
    rng = np.random.default_rng(nsrc + nrec)
    out = []
    for single in (False, True):
        mesh = semgb.Mesh(ex, ey, ez, ex * 10.0, ey * 10.0, ez * 10.0, 1)
        mesh.set_velocity(np.linspace(1500, 3000, mesh.n_elem).astype(np.float32))
        s = semgb.Solver(mesh, 2e-4)
        s.set_sponge(2, 0.1)
        rng = np.random.default_rng(nsrc + nrec)
        s.set_pressure(semgb.LEVEL_CURRENT, rng.standard_normal(mesh.n_nodes).astype(np.float32))
        if nsrc:
            s.set_sources(rng.choice(mesh.n_elem, nsrc), rng.standard_normal((nsrc, 18)).astype(np.float32))
        if nrec:
            s.set_receiver_nodes(rng.choice(mesh.n_nodes, nrec))
        for _ in range(20 if single else 1):
            s.step(1 if single else 20)
        out.append((s.pressure(), s.traces() if nrec else None))
    assert np.array_equal(out[0][0], out[1][0]) and np.abs(out[0][0]).max() > 0
    assert nrec == 0 or np.array_equal(out[0][1], out[1][1])


@pytest.mark.parametrize("nsrc,nrec", [(0, 3), (1, 1), (128, 129), (300, 2000)])
@pytest.mark.parametrize("box", [(32, 21, 33), (17, 64, 16)])
def test_rows_are_the_levels_at_the_receivers(semgb_lib, cuda_device, box, nsrc, nrec):
    """Every row of a run, sampled by the CTAs that found their receivers, against the level read back whole
    after each single step of a second solver without receivers."""
    semgb = semgb_lib
    ex, ey, ez = box
    mesh = semgb.Mesh(ex, ey, ez, ex * 10.0, ey * 10.0, ez * 10.0, 1)
    mesh.set_velocity(np.linspace(1500, 3000, mesh.n_elem).astype(np.float32))
    rng = np.random.default_rng(nsrc + nrec)
    p = rng.standard_normal(mesh.n_nodes).astype(np.float32)
    el, w = rng.choice(mesh.n_elem, nsrc), rng.standard_normal((nsrc, 18)).astype(np.float32)
    # (with the last node of every axis: on far edges of whole tiles plus one node)
    nodes = np.concatenate([rng.choice(mesh.n_nodes, nrec - 1), [mesh.n_nodes - 1]])
    solvers = []
    for receivers in (True, False):
        s = semgb.Solver(mesh, 2e-4)
        s.set_sponge(2, 0.1)
        s.set_pressure(semgb.LEVEL_CURRENT, p)
        if nsrc:
            s.set_sources(el, w)
        if receivers:
            s.set_receiver_nodes(nodes)
        solvers.append(s)
    solvers[0].step(20)
    rows = solvers[0].traces()
    assert rows.shape == (20, nrec)
    for n in range(20):
        solvers[1].step(1)
        assert np.array_equal(rows[n], solvers[1].pressure()[nodes]), n
    assert (np.abs(rows).max(axis=0) > 0).all()
