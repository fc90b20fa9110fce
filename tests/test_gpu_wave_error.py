"""An error of a wave stays until the host reads it after the fit's last tree: the checks in
tests/cpp/wave_error.cu, linked with the library's objects."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_wave_error_outlives_the_next_tree(native, tmp_path):
    from tidegbm_b200 import build

    objs = [os.path.join(build.BUILD, f) for f in sorted(os.listdir(build.BUILD)) if f.endswith(".o")]
    exe = tmp_path / "wave_error"
    subprocess.run([os.path.join(build._cuda_home(), "bin", "nvcc"), "-O1", "-std=c++17", *build.ARCH, "-I", build.CSRC,
                    os.path.join(ROOT, "tests", "cpp", "wave_error.cu"), *objs, "-o", str(exe), "-lpthread"], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    assert out.stdout.strip() == "ok"
