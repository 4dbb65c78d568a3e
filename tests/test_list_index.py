"""The index arithmetic of the step kernels' lists at sizes no test could
hold in memory, on the host."""
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_mid_list_offsets_beyond_31_bits(tmp_path):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    exe = tmp_path / "list_index_check"
    subprocess.run([cxx, "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-o", str(exe),
                    os.path.join(HERE, "native", "list_index_check.cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
    assert "mismatches 0" in out.stdout
