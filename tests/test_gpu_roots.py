"""The short square roots and reciprocals of the FP64 pair kernels against extended precision, over every exponent."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def test_roots_and_reciprocals(tmp_path):
    from fdps_sph_gb300 import build
    exe = tmp_path / "roots_check"
    subprocess.run([build.nvcc(), *build.ARCH, "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    os.path.join(HERE, "cpp", "roots_check.cu"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    print(r.stdout)
    assert r.returncode == 0, r.stdout
