"""The rule that says which host blocks kernels may touch, built as plain C++ with made-up registrations."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))


def test_block_routes(tmp_path):
    exe = tmp_path / "pinned_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", os.path.join(HERE, "cpp", "pinned_check.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
