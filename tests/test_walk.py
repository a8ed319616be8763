"""The item walk's index arithmetic, compiled for the host."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_items_and_reciprocal_division(tmp_path):
    exe = str(tmp_path / "walk")
    subprocess.run([os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc"), "-std=c++17", "-O1", "-arch=sm_100a", "-I" + ROOT,
                    os.path.join(ROOT, "tests", "cpp", "walk.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
