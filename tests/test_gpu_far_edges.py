"""Boxes that are whole tiles plus their last node along x, z or both: that boundary row or column has
no tile of its own and is damped by the last tile's CTAs.  Steps from a random state (boundary
included) against the oracle and, on the same nodes, against the element path; receivers on the far
edges and the corner; batches, groups and the adjoint's forward run against the plain pass bit for
bit; the square order-4 tile."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu

# tile (nodes along x, z) per order
TILES = {1: (16, 16), 2: (32, 16), 3: (48, 12), 4: (64, 16), 5: (40, 20)}


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _case(semgb, order, xt, zt, sponge, tile=None):
    """xt, zt: whole tiles along the axis, or 0 for a ragged size."""
    tx, tz = tile or TILES[order]
    ex = xt * tx // order if xt else tx // order + 2
    ez = zt * tz // order if zt else tz // order + 1
    ey = 7
    n = (ey * order + 1, ez * order + 1, ex * order + 1)
    rng = np.random.default_rng(order + 10 * xt + 100 * zt)
    vel = rng.uniform(1500, 3000, ex * ey * ez).astype(np.float32)
    i = [np.arange(m) for m in n]
    p = (np.sin(0.31 * i[0] + 0.4)[:, None, None] * np.cos(0.23 * i[1])[None, :, None]
         * np.sin(0.19 * i[2] + 0.7)[None, None, :]).astype(np.float32).reshape(-1)
    q = (0.9 * p).astype(np.float32)
    sp = tuple(rng.uniform(0.9, 1.0, m).astype(np.float32) for m in (n[2], n[0], n[1])) if sponge else None
    node = lambda x, z, y: x + n[2] * (z + n[1] * y)  # noqa: E731
    rec = np.array([node(n[2] - 1, 3, 4), node(5, n[1] - 1, 6), node(n[2] - 1, n[1] - 1, n[0] - 2), node(2, 2, 2),
                    node(n[2] - 2, n[1] - 2, 3)])
    from semgb import workloads as W
    dt = W.cfl_dt(10.0, order, 3000.0)
    return (ex, ey, ez), vel, p, q, sp, rec, dt


def _solver(semgb, box, order, vel, p, q, sp, rec, dt):
    mesh = semgb.Mesh(*box, *[10.0 * e for e in box], order)
    mesh.set_velocity(vel)
    s = semgb.Solver(mesh, dt)
    if sp:
        s.set_sponge_profile(*sp)
    s.set_receiver_nodes(rec)
    s.set_pressure(semgb.LEVEL_CURRENT, p)
    s.set_pressure(semgb.LEVEL_PREVIOUS, q)
    return mesh, s


@pytest.mark.parametrize("sponge", [False, True])
@pytest.mark.parametrize("xt,zt", [(1, 1), (2, 0), (0, 2), (1, 3)])
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
def test_whole_tiles_plus_one_node(semgb_lib, cuda_device, order, xt, zt, sponge):
    semgb = semgb_lib
    box, vel, p, q, sp, rec, dt = _case(semgb, order, xt, zt, sponge)
    P = O.Problem(*box, order, *[10.0 * e for e in box], dt, 5, vel, np.zeros(0, np.int64), np.zeros((0, 5), np.float32),
                  rec_node=rec, sponge32=sp)
    want = O.run(P, p, q)
    mesh, s = _solver(semgb, box, order, vel, p, q, sp, rec, dt)
    s.step(5)
    assert rel_l2(s.pressure(semgb.LEVEL_CURRENT), want[0]) <= 1e-5
    assert rel_l2(s.pressure(semgb.LEVEL_PREVIOUS), want[1]) <= 1e-5
    assert rel_l2(s.traces(), want[2]) <= 1e-5
    # the boundary nodes exactly: the stored previous level, damped twice per step
    n = (box[1] * order + 1, box[2] * order + 1, box[0] * order + 1)
    on = np.ones(n, bool)
    on[1:-1, 1:-1, 1:-1] = False
    _, e = _solver(semgb, box, order, vel, p, q, sp, rec, dt)
    e.set_kernel(semgb.KERNEL_ELEMENT)
    e.step(5)
    a, b = s.pressure().reshape(n)[on], e.pressure().reshape(n)[on]
    # (the two paths multiply the three factors in a different order)
    assert np.all(np.abs(a - b) <= 5e-6 * np.abs(b)) and (sponge or np.array_equal(a, b))


@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_batch_group_adjoint_on_whole_tiles(semgb_lib, cuda_device, order):
    semgb = semgb_lib
    box, vel, p, q, sp, rec, dt = _case(semgb, order, 2, 2, True)
    z = np.zeros_like(p)
    src = np.array([box[0] // 2 + (box[2] // 2) * box[0] + 3 * box[0] * box[2], 1 + box[0] + box[0] * box[2]])
    wav = np.random.default_rng(3).standard_normal((2, 40)).astype(np.float32)
    plain = []
    for k in range(2):
        mesh, s = _solver(semgb, box, order, vel, z, z, sp, rec, dt)
        s.set_sources(src[k:k + 1], wav[k:k + 1])
        s.step(40)
        plain.append((s.traces(), s.pressure()))
    assert np.abs(plain[0][0]).max() > 0
    b = semgb.Batch(mesh, dt, 2)
    b.set_sponge_profile(*sp)
    b.set_sources(src, wav)
    b.set_receiver_nodes(rec)
    b.step(40)
    for k in range(2):
        assert np.array_equal(b.traces()[:, :, k], plain[k][0]) and np.array_equal(b.pressure(k), plain[k][1])
    members = [_solver(semgb, box, order, vel, z, z, sp, rec, dt) for _ in range(2)]
    for k, (_, s) in enumerate(members):
        s.set_sources(src[k:k + 1], wav[k:k + 1])
    g = semgb.Group([s for _, s in members])
    g.step(40)
    g.synchronize()
    assert g.launch == semgb.GROUP_ONE_LAUNCH
    for k, (_, s) in enumerate(members):
        assert np.array_equal(s.traces(), plain[k][0]) and np.array_equal(s.pressure(), plain[k][1])
    g.close()
    a = semgb.Adjoint(mesh, dt, 40, 13)
    a.set_sponge_profile(*sp)
    a.set_sources(src[1:], wav[1:])  # next to one of the receivers
    a.set_receiver_nodes(rec)
    assert np.array_equal(a.forward(), plain[1][0])
    grad = a.backward(np.random.default_rng(4).standard_normal((40, len(rec))).astype(np.float32))
    n = (box[1] * order + 1, box[2] * order + 1, box[0] * order + 1)
    assert np.isfinite(grad).all() and np.abs(grad).max() > 0
    assert np.all(grad.reshape(n)[:, -1, :] == 0) and np.all(grad.reshape(n)[:, :, -1] == 0)


def test_square_tile_on_whole_tiles(semgb_lib, cuda_device):
    semgb = semgb_lib
    box, vel, p, q, sp, rec, dt = _case(semgb, 4, 2, 2, True, tile=(32, 32))
    out = []
    for shape in (semgb.TILE_DEFAULT, semgb.TILE_SQUARE):
        _, s = _solver(semgb, box, 4, vel, p, q, sp, rec, dt)
        s.set_tile_shape(shape)
        s.step(9)
        assert s.tile_shape == shape
        out.append((s.pressure(), s.pressure(1), s.traces()))
    assert all(np.array_equal(a, b) for a, b in zip(*out))
