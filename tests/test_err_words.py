"""The error words that kernels set and calls read, one a model (host logic, no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_errors_stay_with_their_model(tmp_path):
    exe = str(tmp_path / "test_err_words")
    subprocess.run([os.environ.get("TI_HOST_CXX", "/usr/bin/g++"), "-std=c++17", "-O1", "-o", exe, os.path.join(ROOT, "tests", "cpp", "test_err_words.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
