"""The row of a mode in the update kernel (mode_row of csrc/mode_index.cuh, as k_rk_update calls
it), for every mode q of the largest plane that a z length can meet."""
import os
import shutil
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_row_of_a_mode(tmp_path):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    exe = tmp_path / "mode_index_test"
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "pandora-2.0_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "mode_index_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == "23 lengths OK"
