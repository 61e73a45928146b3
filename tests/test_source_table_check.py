"""The pass that adds the next step's sources refuses, before it launches, a source table with an array
missing that its kernel would read: the single-shot kernel reads the grouping and the owning CTAs, the
many-shot kernel neither.  No GPU is needed: the refusal comes before any CUDA call."""
import os
import shutil
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include "stencil.h"
using namespace semgb;
int main()
{
    // stands for any array; never dereferenced on the host, and every call below is refused
    static float any_f; static int any_i; static int64_t any_l;
    const SourceTable full{&any_l, &any_f, &any_f, &any_i, &any_i, 1, 4};
    int bad = 0;
    for (int order = 1; order <= 5; order++)
        for (int nshot : {1, 2})
            for (int missing = 0; missing < 6; missing++) {
                if (nshot > 1 && missing >= 3) continue;  // not read by the many-shot kernel
                StencilTables t;
                t.order = order;
                t.nshot = nshot;
                StencilArgs a{};
                a.inject = 1;
                a.src = full;
                a.src_cta = &any_i;
                if (missing == 0) a.src.node = nullptr;
                if (missing == 1) a.src.coef = nullptr;
                if (missing == 2) a.src.wavelet = nullptr;
                if (missing == 3) a.src.off = nullptr;
                if (missing == 4) a.src.perm = nullptr;
                if (missing == 5) a.src_cta = nullptr;
                if (launch_stencil(t, a, 0, false, nullptr) != cudaErrorInvalidValue) bad++;
            }
    return bad;
}
"""


def test_incomplete_source_table_is_refused(semgb_lib, tmp_path):
    sys.path.insert(0, os.path.join(ROOT, "proxy-geos-hc_gb300"))
    import build
    cuda = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    src, exe = tmp_path / "p.cpp", tmp_path / "p"
    src.write_text(PROGRAM)
    lib_dir = os.path.dirname(build.LIB)
    r = subprocess.run(["g++", "-std=c++17", "-I", build.CSRC, "-I", cuda, str(src), "-o", str(exe), "-L", lib_dir, "-lsemgb",
                        f"-Wl,-rpath,{lib_dir}"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-2000:]
    # hidden devices: on a machine with a GPU a launch that is not refused must not run either
    r = subprocess.run([str(exe)], env={**os.environ, "CUDA_VISIBLE_DEVICES": ""}, timeout=60)
    assert r.returncode == 0
