"""Node planes at the far end of the float range (host code, no GPU)."""
import os
import shutil
import subprocess

from conftest import ROOT


def test_lo_planes_beyond_the_largest_float(tmp_path):
    exe = str(tmp_path / "node_planes_far")
    src = os.path.join(ROOT, "tests", "c", "node_planes_far.cpp")
    subprocess.run([shutil.which("g++") or "g++", "-std=c++17", "-O2", "-ffp-contract=off", src, "-o", exe], check=True)
    p = subprocess.run([exe], capture_output=True, text=True)
    assert p.returncode == 0 and p.stdout == "ok\n", p.stdout
