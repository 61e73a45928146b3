"""The streaming call (samples handed to the source launch by value, receiver rows written to pinned
memory by the device) gives the bits of the same run with the wavelets stored: source counts around
the by-value limit of 32, receiver rows on both sides of the pinned buffer's 16384 values, calls of
one step and around the graph length, before and after a reset."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nsrc,nrec", [(1, 1), (3, 16), (32, 1024), (33, 1025), (2, 16385)])
def test_streaming_equals_stored(semgb_lib, cuda_device, nsrc, nrec):
    semgb = semgb_lib
    from semgb import workloads as W
    chunks = [1, 1, 16, 1, 17, 2, 1]
    n = sum(chunks)
    wl = W.small_random(9, 8, 7, 2, n, seed=nsrc, nsrc=nsrc, nrec=nrec)
    wl.src_xyz[-1] = wl.src_xyz[0]  # two sources in one element
    mesh, s = semgb.solver_from_workload(wl)
    s.step(n)
    want, field = s.traces(), s.pressure()
    assert np.abs(want).max() > 0
    wav = np.stack([semgb.ricker(n, wl.dt, float(f), wl.ricker_order) for f in wl.f0])
    mesh2, s2 = semgb.solver_from_workload(wl)
    s2.set_source_points(wl.src_xyz, np.zeros_like(wav))  # every sample comes from the calls
    for _ in range(2):
        k = 0
        for c in chunks:
            out = np.full((c, nrec), np.nan, np.float32)
            s2.step_host(c, np.ascontiguousarray(wav[:, k:k + c].T), out)
            assert np.array_equal(out, want[k:k + c])
            k += c
        assert np.array_equal(s2.traces(), want) and np.array_equal(s2.pressure(), field)
        s2.reset()
        assert not s2.pressure().any() and s2.steps_done == 0
    with pytest.raises(semgb.SemError):
        s2.step_host(n + 1, np.zeros((n + 1, nsrc), np.float32))
