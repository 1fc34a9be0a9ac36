"""The row of a mode in the update kernel (mode_row of csrc/mode_index.cuh, as k_rk_update calls
it), for every mode q of the largest plane that a z length can meet."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LENGTHS = sorted(2 ** a * f for a in range(3, 11) for f in (1, 3, 5, 7) if 16 <= 2 ** a * f <= 1024)


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    exe = tmp_path_factory.mktemp("mode_index") / "mode_index_test"
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "pandora-2.0_b200", "csrc"),
                    os.path.join(ROOT, "tests", "native", "mode_index_test.cpp"), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("nz", LENGTHS)
def test_row_of_a_mode(harness, nz):
    r = subprocess.run([harness, str(nz)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.strip() == f"{(2 * (1024 // 3) + 1) * (2 * (nz // 3) + 1)} modes OK"
