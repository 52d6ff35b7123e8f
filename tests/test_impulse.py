"""CPU check of the solver's accumulate/clamp loop without clamps: tests/impulse_check.cpp compiles
the kernels' own header (nans_projekat_gb300/csrc/nans_impulse.cuh) for the host and compares the
last round's differences bit for bit with the loop of Constraint (code/nans.cpp:1176-1230) wherever
the header decides, over seeded increments that include ones near the limits of its two cases."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_direct_impulse_equals_the_loop(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    exe = str(tmp_path / "impulse_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off",
                    "-I", os.path.join(ROOT, "nans_projekat_gb300", "csrc"),
                    os.path.join(ROOT, "tests", "impulse_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    ok, decided, tried = r.stdout.split()
    assert ok == "ok" and int(decided) > int(tried) // 2
