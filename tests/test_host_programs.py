"""Host logic of the library's sources, checked by small C++ programs (``tests/host``)
that are compiled against its headers; each prints a line per failure."""
import os
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "hssmatrices.jl_gb300", "csrc")
LIB = os.path.join(ROOT, "hssmatrices.jl_gb300", "lib")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def run(tmp_path, name, link):
    exe = str(tmp_path / name)
    cmd = ["g++", "-std=c++17", "-O1", "-I", CSRC, "-I", os.path.join(ROOT, "include"),
           "-I", os.path.join(CUDA, "include"), os.path.join(ROOT, "tests", "host", name + ".cpp"), "-o", exe]
    if link:
        cmd += ["-L", LIB, "-lhssgpu", "-Wl,-rpath," + LIB, "-L", os.path.join(CUDA, "lib64"), "-lcudart",
                "-Wl,-rpath," + os.path.join(CUDA, "lib64")]
    built = subprocess.run(cmd, capture_output=True, text=True)
    assert built.returncode == 0, built.stderr
    out = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0 and out.stdout == "", out.stdout + out.stderr


@pytest.mark.parametrize("name", ["levels_split", "levels_key"])
def test_linked(lib, tmp_path, name):
    run(tmp_path, name, link=True)


@pytest.mark.parametrize("name", ["smem_opt_in", "recip"])
def test_alone(tmp_path, name):
    run(tmp_path, name, link=False)


def test_no_process_wide_opt_in():
    """The attribute of more than 48 KB of shared memory is set per device: by the opt-in
    objects, or on every call."""
    for f in sorted(os.listdir(CSRC)):
        lines = open(os.path.join(CSRC, f)).read().splitlines()
        for i, line in enumerate(lines):
            if "cudaFuncSetAttribute(" in line:
                assert not any("static bool" in x for x in lines[max(0, i - 4):i]), f"{f}:{i + 1}"
