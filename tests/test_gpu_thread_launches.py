"""Plans of two host threads that run the same kernels with different amounts of shared
memory.  The limit on it is one value per kernel, so the library must never set it to what
one plan needs; Python's threads seldom meet there, so the caller is a C++ program."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("no CUDA device", allow_module_level=True)


def test_no_launch_fails(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = os.path.join(str(tmp_path), "thread_launches")
    libdir = os.path.join(ROOT, "recon_b200")
    subprocess.run([nvcc, "-std=c++17", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "thread_launches.cpp"), "-o", exe, "-L", libdir,
                    "-lrecon_b200", "-Xlinker", f"-rpath={libdir}"], check=True)
    res = subprocess.run([exe, "30000"], capture_output=True, text=True, timeout=600)
    assert res.returncode == 0, res.stdout + res.stderr
