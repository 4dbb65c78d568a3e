"""The on-the-fly coefficients' reciprocal, phase and Lagrange weights, the
kernels' own source compiled for the host, against binary128."""
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_pieces_of_the_coefficients_keep_their_bounds(tmp_path):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    exe = tmp_path / "coef_check"
    subprocess.run([cxx, "-std=gnu++17", "-O2", "-ffp-contract=off", "-w", "-I/usr/local/cuda/include", "-o",
                    str(exe), os.path.join(HERE, "native", "coef_check.cpp"), "-lquadmath"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout
    assert "mismatches 0" in out.stdout
