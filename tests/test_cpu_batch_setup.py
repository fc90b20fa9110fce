"""The set-ups of a batched fit side by side, and one after another where the device has no room for
that (tidegbm_b200/csrc/batch_setup.h, host only): the checks in tests/cpp/test_batch_setup.cpp."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_batch_setup(tmp_path):
    exe = tmp_path / "test_batch_setup"
    subprocess.run(["g++", "-O1", "-std=c++17", "-pthread", "-Wall", "-I", os.path.join(ROOT, "tidegbm_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_batch_setup.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    assert out.stdout.strip() == "ok"
