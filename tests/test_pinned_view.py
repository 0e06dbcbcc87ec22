"""Which host arrays the layout kernels reach themselves: those that lie in
pinned memory from their first to their last byte.  Host code against a
stand-in for the CUDA runtime."""
import subprocess
from pathlib import Path

REPO = Path(__file__).resolve().parent.parent


def test_pinned_view(tmp_path):
    exe = tmp_path / "pinned_view"
    subprocess.run(["g++", "-std=c++17", "-I/usr/local/cuda/include", "-I" + str(REPO / "ipcc2021-final_gb300/csrc"),
                    str(REPO / "tests/cpp/pinned_view.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
