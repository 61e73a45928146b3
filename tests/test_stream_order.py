"""What a handle's kernels read is put in place on the handle's own stream: its non-blocking stream does not
wait for the default stream, where plain copies and fills run, and a plain copy from pageable memory may
return before it has landed.  On the sources (no GPU), and as runs that start at once on fresh handles."""
import glob
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "proxy-geos-hc_gb300", "csrc")


def _code(path):
    src = open(path).read()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", src, flags=re.S))


def test_no_upload_or_fill_on_the_default_stream():
    files = [f for f in sorted(glob.glob(os.path.join(CSRC, "*"))) if f.endswith((".cu", ".cuh", ".h", ".cpp"))]
    assert len(files) > 15
    for f in files:
        code = _code(f)
        for m in re.finditer(r"\bcudaMem(cpy|cpy2D|set)\s*\(", code):
            call = code[m.start():code.index(";", m.start())]
            assert m.group(1) != "set" and "HostToDevice" not in call, (os.path.basename(f), call)
        if "cudaMemcpyToSymbol(" in code:  # on the default stream: waited for after the last one
            assert re.match(r"[^;]*;\s*return cudaStreamSynchronize\(0\);", code[code.rindex("cudaMemcpyToSymbol("):]), f


@pytest.mark.gpu
def test_runs_started_at_once_on_fresh_handles(semgb_lib, cuda_device):
    semgb = semgb_lib
    from semgb import workloads as W
    import torch
    wls = [W.small_random(6 + i % 5, 7, 5 + i % 3, 1 + i % 5, 20, seed=160 + i, nsrc=3, nrec=40) for i in range(10)]
    want = None
    for waited in (True, False, False, False):
        got = []
        for kernel in (semgb.KERNEL_STENCIL, semgb.KERNEL_ELEMENT):
            handles = []
            for w in wls:
                mesh, s = semgb.solver_from_workload(w, kernel)
                if waited:
                    torch.cuda.synchronize()
                s.step(w.nsteps)
                handles.append((mesh, s))
            for _, s in handles:
                s.synchronize()
                got.append((s.traces(), s.pressure()))
            for mesh, s in handles:
                s.close()
                mesh.close()
        want = want or got
        for k, (a, b) in enumerate(zip(got, want)):
            assert np.abs(b[0]).max() > 0
            if k < len(wls):
                assert np.array_equal(a[0], b[0]) and np.array_equal(a[1], b[1])
            else:  # the element path's float atomics have no fixed order
                assert np.abs(a[1] - b[1]).max() <= 1e-5 * np.abs(b[1]).max()
