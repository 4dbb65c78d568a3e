"""The index arithmetic of the step kernels' lists at sizes no test could
hold in memory, and the sizes of the far kernel's partials, on the host."""
import os
import shutil
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def run_native(name, tmp_path):
    cxx = shutil.which("g++") or "/usr/bin/g++"
    exe = tmp_path / name
    subprocess.run([cxx, "-std=c++17", "-O1", "-I/usr/local/cuda/include", "-o", str(exe),
                    os.path.join(HERE, "native", name + ".cpp")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
    assert "mismatches 0" in out.stdout


def test_mid_list_offsets_beyond_31_bits(tmp_path):
    run_native("list_index_check", tmp_path)


def test_partials_of_every_cut_fit(tmp_path):
    run_native("far_parts_check", tmp_path)
