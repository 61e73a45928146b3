"""A run of steps enqueued at once (sources added by the pass before, programmatic dependent
launches, graphs of 16) gives the bits of the same steps enqueued one by one (a source launch each):
counts around the graph length, sources sharing nodes, on tile edges and corners of a box of several
tiles and y-chunks, next to the boundary and outside the wavelet, with and without the boundary
network, batched and grouped."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
COUNTS = [1, 2, 15, 16, 17, 33]


def _wavelet(nsrc, n, seed):
    return np.random.default_rng(seed).standard_normal((nsrc, n)).astype(np.float32)


def _solver(semgb, ex, ey, ez, o, elements, nsamples, variant="default"):
    mesh = semgb.Mesh(ex, ey, ez, ex * 10.0, ey * 10.0, ez * 10.0, o)
    mesh.set_velocity(np.linspace(1500, 3000, mesh.n_elem).astype(np.float32))
    s = semgb.Solver(mesh, 2e-4)
    if variant == "element":
        s.set_kernel(semgb.KERNEL_ELEMENT)
    if variant == "reference":
        s.set_rounding(semgb.ROUNDING_REFERENCE)
    s.set_sponge(1, 0.1)
    s.set_sources(elements, _wavelet(len(elements), nsamples, 3))
    nx, nz = ex * o + 1, ez * o + 1
    src_nodes = [(e % ex) * o + ((e // ex) % ez) * o * nx + (e // (ex * ez)) * o * nx * nz for e in elements]
    s.set_receiver_nodes(np.array(src_nodes + [5, mesh.n_nodes - 1, mesh.n_nodes // 2]))
    return mesh, s


def _elements(ex, ey, ez):
    at = [(0, 0, 0), (1, 1, 1), (ex - 1, ez - 1, ey - 1), (ex // 2, ez // 2, ey // 2), (ex // 2, ez // 2, ey // 2),
          (16 % ex, 4 % ez, 3 % ey), (15 % ex, 5 % ez, 2 % ey), (1, 1, 1), (8 % ex, 8 % ez, ey // 2)]
    return np.array([x + z * ex + y * ex * ez for x, z, y in at])


@pytest.mark.parametrize("order,variant", [(1, "default"), (2, "default"), (3, "default"), (4, "default"),
                                           (5, "default"), (4, "reference")])
def test_run_equals_single_steps(semgb_lib, cuda_device, order, variant):
    semgb = semgb_lib
    ex, ey, ez = {1: (70, 41, 40), 2: (40, 30, 22), 3: (20, 25, 18), 4: (19, 23, 11), 5: (11, 12, 9)}[order]
    el = _elements(ex, ey, ez)
    for n in COUNTS:
        nsamples = n - 1 if n > 2 else n  # the last step has no sample left
        m1, a = _solver(semgb, ex, ey, ez, order, el, nsamples, variant)
        m2, b = _solver(semgb, ex, ey, ez, order, el, nsamples, variant)
        a.step(n)
        for _ in range(n):
            b.step(1)
        assert np.array_equal(a.traces(), b.traces()), n
        assert np.array_equal(a.pressure(), b.pressure()) and np.array_equal(a.pressure(1), b.pressure(1)), n
        assert np.abs(a.pressure()).max() > 0
        for x in (a, b, m1, m2):
            x.close()


@pytest.mark.parametrize("layer", [0, 1])
@pytest.mark.parametrize("deep", [False, True])
def test_corrected_run_equals_single_steps(semgb_lib, cuda_device, layer, deep):
    semgb = semgb_lib
    ex, ey, ez, o = 12, 11, 10, 3
    el = np.array([5 + 5 * ex + 5 * ex * ez]) if deep else _elements(ex, ey, ez)
    net = semgb.Mlp(4)
    for n in COUNTS:
        got = []
        for single in (False, True):
            m, s = _solver(semgb, ex, ey, ez, o, el, n)
            abc = semgb.Abc(s, net, layer)
            for k in [1] * n if single else [n]:
                abc.step(k)
            got.append((s.traces(), s.pressure(), s.pressure(1)))
            for x in (abc, s, m):
                x.close()
        assert all(np.array_equal(a, b) for a, b in zip(*got)), n


@pytest.mark.parametrize("order", [1, 2, 3, 4, 5])
def test_batch_run_equals_single_steps(semgb_lib, cuda_device, order):
    semgb = semgb_lib
    ex, ey, ez = {1: (40, 21, 20), 2: (30, 20, 12), 3: (20, 15, 10), 4: (18, 13, 9), 5: (11, 9, 8)}[order]
    mesh = semgb.Mesh(ex, ey, ez, ex * 10.0, ey * 10.0, ez * 10.0, order)
    mesh.set_velocity(np.linspace(1500, 3000, mesh.n_elem).astype(np.float32))
    el = _elements(ex, ey, ez)[:7].copy()
    el[2] = -1  # a shot without a source
    for n in COUNTS:
        got = []
        for single in (False, True):
            b = semgb.Batch(mesh, 2e-4, len(el))
            b.set_sources(el, _wavelet(len(el), n, 5))
            b.set_receiver_nodes(np.array([3, mesh.n_nodes // 2, mesh.n_nodes // 2 + 1]))
            for k in [1] * n if single else [n]:
                b.step(k)
            got.append([b.traces()] + [b.pressure(i) for i in range(len(el))])
            b.close()
        assert all(np.array_equal(x, y) for x, y in zip(*got)), n
    mesh.close()


@pytest.mark.parametrize("launch", [0, 1])
def test_group_run_equals_solo_single_steps(semgb_lib, cuda_device, launch):
    semgb = semgb_lib
    boxes = [(9, 8, 7, 2), (6, 14, 5, 3), (19, 6, 5, 4), (30, 9, 8, 1)]
    for n in COUNTS:
        members = [_solver(semgb, ex, ey, ez, o, _elements(ex, ey, ez), n) for ex, ey, ez, o in boxes]
        solo = [_solver(semgb, ex, ey, ez, o, _elements(ex, ey, ez), n) for ex, ey, ez, o in boxes]
        g = semgb.Group([s for _, s in members], launch)
        g.step(n)
        g.synchronize()
        for (_, a), (_, b) in zip(members, solo):
            for _ in range(n):
                b.step(1)
            assert np.array_equal(a.traces(), b.traces()) and np.array_equal(a.pressure(), b.pressure()), n
        g.close()
        for m, s in members + solo:
            s.close()
            m.close()


@pytest.mark.parametrize("calls", [[1], [2], [3], [15], [16], [17], [33], [16] * 9 + [3], [145, 18]])
def test_element_run_equals_single_steps(semgb_lib, cuda_device, calls):
    """The element path's steps: alone, in pairs and in runs of 16 replayed from graphs.  Its float atomics add
    the eight or fewer contributions of a node in any order: a few units in the last place per step."""
    semgb = semgb_lib
    ex, ey, ez, order = 7, 8, 6, 3
    el, n = _elements(ex, ey, ez), sum(calls)
    m1, a = _solver(semgb, ex, ey, ez, order, el, n, "element")
    m2, b = _solver(semgb, ex, ey, ez, order, el, n, "element")
    for c in calls:
        a.step(c)
    for _ in range(n):
        b.step(1)
    for x, y in ((a.traces(), b.traces()), (a.pressure(), b.pressure()), (a.pressure(1), b.pressure(1))):
        assert np.abs(x - y).max() <= 1e-5 * np.abs(y).max()
    assert np.abs(a.pressure()).max() > 0
    for x in (a, b, m1, m2):
        x.close()


@pytest.mark.parametrize("members", [16, 17])
def test_branches_of_few_steps_equal_solo_single_steps(semgb_lib, cuda_device, members):
    """Calls of two to four steps, which more than 16 branches replay in pairs, from both parities, and of five."""
    semgb = semgb_lib
    boxes = [(3 + i % 4, 4, 3 + i % 3, 1 + i % 4) for i in range(members)]
    calls = [2, 3, 2, 1, 3, 4, 5, 18, 20, 21]
    n = sum(calls)
    grouped = [_solver(semgb, ex, ey, ez, o, _elements(ex, ey, ez) % (ex * ey * ez), n) for ex, ey, ez, o in boxes]
    solo = [_solver(semgb, ex, ey, ez, o, _elements(ex, ey, ez) % (ex * ey * ez), n) for ex, ey, ez, o in boxes]
    g = semgb.Group([s for _, s in grouped], semgb.GROUP_BRANCHES)
    for c in calls:
        g.step(c)
    g.synchronize()
    for (_, a), (_, b) in zip(grouped, solo):
        for _ in range(n):
            b.step(1)
        assert np.array_equal(a.traces(), b.traces()) and np.array_equal(a.pressure(), b.pressure())
        assert np.abs(b.traces()).max() > 0
    g.close()
    for m, s in grouped + solo:
        s.close()
        m.close()
