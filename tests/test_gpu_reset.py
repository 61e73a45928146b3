"""sem_solver_reset and sem_abc_reset are ordered with the steps around them: a run started at once
after a reset (no synchronisation between) gives the bits of a run of a fresh handle.  Many small
members make the reset longer than the time to enqueue the first step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_group_steps_right_after_reset(semgb_lib, cuda_device):
    semgb = semgb_lib
    from semgb import workloads as W
    wls = [W.small_random(6 + i % 5, 7, 5 + i % 3, 2 + i % 3, 24, seed=60 + i, nsrc=1, nrec=8) for i in range(24)]
    members = [semgb.solver_from_workload(w, semgb.KERNEL_STENCIL) for w in wls]
    solvers = [s for _, s in members]
    g = semgb.Group(solvers)
    g.step(24)
    g.synchronize()
    want = [s.traces() for s in solvers]
    assert all(np.abs(t).max() > 0 for t in want)
    for _ in range(3):
        for s in solvers:
            s.reset()
        g.step(24)
        g.synchronize()
        for s, t in zip(solvers, want):
            assert np.array_equal(s.traces(), t)
    g.close()


@pytest.mark.parametrize("network", [False, True])
def test_solver_steps_right_after_reset(semgb_lib, cuda_device, network):
    semgb = semgb_lib
    from semgb import workloads as W
    wl = W.small_random(40, 38, 36, 4, 12, seed=91, nsrc=1, nrec=16)  # a reset of tens of microseconds
    mesh, s = semgb.solver_from_workload(wl, semgb.KERNEL_STENCIL)
    net = semgb.Mlp(2)
    abc = semgb.Abc(s, net, 0) if network else None
    want = None
    for _ in range(4):
        (abc if network else s).step(12)
        got = (s.traces(), s.pressure())
        want = want or got
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
        s.reset()
        if network:
            abc.reset()
    assert np.abs(want[1]).max() > 0
