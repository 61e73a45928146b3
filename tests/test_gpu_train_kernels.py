"""Training kernels of the boundary network at the sizes where their split of the work changes: one
row, parts of a 16-row group and of a 128-row tile, the switch of rows and units per CTA (4864
rows), more rows than one round of partial-sum slots (77,824), and the adjoint's pass over more
boundary nodes than one round.  Gradients against the oracle (tolerances of test_gpu_abc.py) and
central differences."""
import numpy as np
import pytest

from oracle import mlp_oracle as M

pytestmark = pytest.mark.gpu


def rel_l2(a, b):
    a, b = np.asarray(a, np.float64), np.asarray(b, np.float64)
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("n", [1, 15, 17, 128, 129, 4864, 4865, 77824, 77824 + 130])
def test_gradient_row_counts(semgb_lib, cuda_device, n):
    semgb = semgb_lib
    rng = np.random.default_rng(n)
    p = (rng.standard_normal(M.N_PARAMS) * 0.2).astype(np.float32)
    x = rng.uniform(-1, 1, (n, 81)).astype(np.float32)
    t = rng.standard_normal(n).astype(np.float32)
    net = semgb.Mlp(1)
    net.params = p
    loss, g = net.loss_grad(x, t)
    lo, go = M.loss_grad(p, x, t)
    assert abs(loss - lo) <= 2e-3 * lo
    o = 0
    for size in (64 * 81, 64, 64 * 64, 64, 64, 1):
        assert rel_l2(g[o:o + size], go[o:o + size]) < 5e-3, (o, size)
        o += size
    # a second pass with fewer rows on the same handle reuses the larger work arrays
    m = max(1, n // 3)
    _, g2 = net.loss_grad(x[:m], t[:m])
    assert rel_l2(g2, M.loss_grad(p, x[:m], t[:m])[1]) < 5e-3
    net.close()


def test_adjoint_over_two_rounds_of_boundary_nodes(semgb_lib, cuda_device):
    semgb = semgb_lib
    from semgb import workloads as W
    ne, o, h, c, steps = 58, 2, 10.0, 2000.0, 14
    mesh = semgb.Mesh(ne, ne, ne, ne * h, ne * h, ne * h, o)
    mesh.set_velocity(np.full(ne ** 3, c, np.float32))
    s = semgb.Solver(mesh, W.cfl_dt(h, o, c))
    s.set_kernel(semgb.KERNEL_STENCIL)
    n = ne * o + 1
    wav = np.sin(np.arange(steps) * 0.5)[None].astype(np.float32)
    s.set_sources(np.array([(ne - 2) + (ne - 2) * ne + (ne - 2) * ne * ne]), wav)  # in the last corner
    net = semgb.Mlp(3)
    rng = np.random.default_rng(11)
    p0 = (rng.standard_normal(M.N_PARAMS) * 0.02).astype(np.float32)
    net.params = p0
    abc = semgb.Abc(s, net, 0)
    assert abc.n_nodes > 77824
    i = np.arange(n - 9, n)
    roi = (i[:, None, None] * n * n + i[None, :, None] * n + i[None, None, :]).reshape(-1)
    ref = np.zeros((steps, len(roi)), np.float32)
    loss, g = abc.bptt(roi, ref)
    assert loss > 0 and np.all(np.isfinite(g))
    h1 = 64 * 81
    fp32 = np.r_[np.arange(h1, h1 + 64), np.arange(h1 + 64 + 4096, len(p0))]
    for _ in range(2):
        v = np.zeros_like(p0)
        v[fp32] = rng.standard_normal(len(fp32)).astype(np.float32)
        lp = []
        for sign in (1.0, -1.0):
            net.params = p0 + np.float32(sign * 1e-2) * v
            lp.append(abc.bptt(roi, ref, grad=False)[0])
        net.params = p0
        fd = (lp[0] - lp[1]) / 2e-2
        ad = float(np.dot(g.astype(np.float64), v.astype(np.float64)))
        assert abs(fd - ad) <= 2e-2 * abs(fd), (fd, ad)
    for x in (abc, net, s, mesh):
        x.close()


@pytest.mark.parametrize("twice", [False, True])
def test_adjoint_step_groups_and_repeated_region_nodes(semgb_lib, cuda_device, twice):
    """The adjoint sums the parameter gradients of several steps at once: on a 3^3 order-2 box (2 tiles
    of boundary nodes, 304 steps per group) 310 steps take two groups, 304 exactly one, each against
    central differences; and a region of interest that lists nodes twice counts them twice."""
    semgb = semgb_lib
    from semgb import workloads as W
    ne, o, h, c = 3, 2, 10.0, 2000.0
    for steps in (304, 310):
        mesh = semgb.Mesh(ne, ne, ne, ne * h, ne * h, ne * h, o)
        mesh.set_velocity(np.full(ne ** 3, c, np.float32))
        s = semgb.Solver(mesh, W.cfl_dt(h, o, c))
        s.set_kernel(semgb.KERNEL_STENCIL)
        s.set_sponge(1, 0.1)
        wav = np.exp(-((np.arange(steps) - (steps - 14)) / 4.0) ** 2)[None].astype(np.float32)  # late pulse
        s.set_sources(np.array([1 + ne + ne * ne]), wav)
        net = semgb.Mlp(3)
        rng = np.random.default_rng(13)
        p0 = (rng.standard_normal(M.N_PARAMS) * 0.02).astype(np.float32)
        net.params = p0
        abc = semgb.Abc(s, net, 0)
        roi = np.arange(100, 200)
        if twice:
            roi = np.concatenate([roi, roi[::-1]])
        ref = np.zeros((steps, len(roi)), np.float32)
        loss, g = abc.bptt(roi, ref)
        assert loss > 0 and np.all(np.isfinite(g))
        if twice:
            l1, g1 = abc.bptt(roi[:100], ref[:, :100])
            assert abs(loss - 2 * l1) <= 1e-6 * loss and rel_l2(g, 2 * g1) < 1e-4
        h1 = 64 * 81
        fp32 = np.r_[np.arange(h1, h1 + 64), np.arange(h1 + 64 + 4096, len(p0))]
        v = np.zeros_like(p0)
        v[fp32] = rng.standard_normal(len(fp32)).astype(np.float32)
        lp = []
        for sign in (1.0, -1.0):
            net.params = p0 + np.float32(sign * 1e-2) * v
            lp.append(abc.bptt(roi, ref, grad=False)[0])
        fd = (lp[0] - lp[1]) / 2e-2
        ad = float(np.dot(g.astype(np.float64), v.astype(np.float64)))
        assert abs(fd - ad) <= 2e-2 * abs(fd), (steps, fd, ad)
        for x in (abc, net, s, mesh):
            x.close()
