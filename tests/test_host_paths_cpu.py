"""Host paths of the library (copies, opt-ins, kept buffers, status words) on a CUDA runtime without a GPU.

The library's own objects are linked with tests/shim/fake_cudart.cpp in place
of cudart; each case is a run of that program.  Freed host memory is filled
with a pattern (MALLOC_PERTURB_), so that a copy from it shows.
"""
import os
import subprocess

import pytest

from conftest import ROOT

SHIM = os.path.join(ROOT, "tests", "shim")


@pytest.fixture(scope="module")
def program(pg, tmp_path_factory):
    cuda = next((c for c in (os.environ.get("CUDA_HOME"), "/usr/local/cuda") if c and os.path.isdir(c)), None)
    if cuda is None:
        pytest.skip("CUDA toolkit headers not found")
    exe = str(tmp_path_factory.mktemp("host") / "host_paths")
    folder = os.path.join(ROOT, "pisces-1_gb300")
    objs = [os.path.join(folder, "_build", f + ".o") for f in sorted(os.listdir(os.path.join(folder, "csrc")))
            if f.endswith((".cu", ".cpp"))]
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", SHIM, "-I", os.path.join(ROOT, "include"),
                    "-I", os.path.join(cuda, "include"), os.path.join(SHIM, "host_paths.cpp"),
                    os.path.join(SHIM, "fake_cudart.cpp"), *objs, "-o", exe, "-lpthread",
                    "-Wl,--unresolved-symbols=ignore-all"], check=True)
    return exe


@pytest.mark.parametrize("case", ["scpol_upload", "hx_status", "hx_captured", "second_device", "potential_tables", "slice_grids",
                                  "kept_buffers", "captured_counters"])
def test_host_path(program, case):
    r = subprocess.run([program, case], env=dict(os.environ, MALLOC_PERTURB_="165"), capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
