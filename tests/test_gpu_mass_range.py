"""The discrete problem does not depend on the element size when dt scales with it: boxes of 10 m,
10^14 m (masses above the float range) and 10^-14 m elements (below it) give the same fields and,
scaled, the same adjoint gradient (a double quotient per node rounded to float) up to rounding, for
velocity and slowness models; rounding differs per size (the sizes are not powers of two apart):
2e-5 after 30 steps."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 3, 5])
@pytest.mark.parametrize("model", ["velocity", "slowness"])
def test_fields_do_not_depend_on_the_length_unit(semgb_lib, cuda_device, order, model):
    semgb = semgb_lib
    from semgb import workloads as W
    ex, ey, ez = 5, 4, 6
    rng = np.random.default_rng(order)
    vel = rng.uniform(1500, 3000, ex * ey * ez).astype(np.float32)
    n = (ey * order + 1) * (ez * order + 1) * (ex * order + 1)
    m = (1.0 / rng.uniform(1500, 3000, n) ** 2).astype(np.float32)
    p = rng.standard_normal(n).astype(np.float32)
    out = []
    for h in (10.0, 1e14, 1e-14):
        mesh = semgb.Mesh(ex, ey, ez, ex * h, ey * h, ez * h, order)
        if model == "velocity":
            mesh.set_velocity(vel)
        else:
            mesh.set_slowness2(m)
        s = semgb.Solver(mesh, W.cfl_dt(h, order, 3000.0))
        s.set_sponge(1, 0.1)
        s.set_pressure(semgb.LEVEL_CURRENT, p)
        s.set_pressure(semgb.LEVEL_PREVIOUS, p)
        s.step(30)
        out.append(s.pressure().astype(np.float64))
        s.close()
        mesh.close()
    assert np.linalg.norm(out[0]) > 0
    for o in out[1:]:
        assert np.linalg.norm(o - out[0]) <= 2e-5 * np.linalg.norm(out[0])


@pytest.mark.parametrize("model", ["velocity", "slowness"])
def test_gradient_does_not_depend_on_the_length_unit(semgb_lib, cuda_device, model):
    """dL/dm for a given residual and unit source coefficient: with dt ~ h the source term and the
    traces scale with h^2 (dt^2 c^2) and so does the gradient."""
    semgb = semgb_lib
    from semgb import workloads as W
    ex, ey, ez, order, steps = 6, 5, 7, 3, 40
    rng = np.random.default_rng(8)
    vel = rng.uniform(1500, 3000, ex * ey * ez).astype(np.float32)
    n = (ey * order + 1) * (ez * order + 1) * (ex * order + 1)
    m = (1.0 / rng.uniform(1500, 3000, n) ** 2).astype(np.float32)
    nodes = rng.choice(n, 12, replace=False)
    res = rng.standard_normal((steps, 12)).astype(np.float32)
    wav = rng.standard_normal((1, steps)).astype(np.float32)
    out = []
    for h in (10.0, 1e5, 1e-5):
        mesh = semgb.Mesh(ex, ey, ez, ex * h, ey * h, ez * h, order)
        mesh.set_velocity(vel)
        if model == "slowness":
            mesh.set_slowness2(m)
        a = semgb.Adjoint(mesh, W.cfl_dt(h, order, 3000.0), steps, 15)
        a.set_sponge(1, 0.1)
        a.set_sources(np.array([2 + 2 * ex + 2 * ex * ez]), wav)
        a.set_receiver_nodes(nodes)
        a.forward()
        out.append(a.backward(res).astype(np.float64) / (h / 10.0) ** 2)
        a.close()
        mesh.close()
    assert np.linalg.norm(out[0]) > 0
    for o in out[1:]:
        assert np.linalg.norm(o - out[0]) <= 2e-5 * np.linalg.norm(out[0])
