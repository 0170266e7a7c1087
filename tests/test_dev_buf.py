"""The owning device buffer (host code, no GPU)."""
import os
import shutil
import subprocess

from conftest import ROOT
from cudart_gb300.build import CUDA_HOME


def test_a_failed_allocation_leaves_an_empty_buffer(tmp_path):
    exe = str(tmp_path / "dev_buf")
    src = os.path.join(ROOT, "tests", "c", "dev_buf.cpp")
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-O1", "-I" + os.path.join(CUDA_HOME, "include"), src,
                    "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True)
    assert p.returncode == 0 and p.stdout == "ok\n", p.stdout
