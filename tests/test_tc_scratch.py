"""The tensor-core kernels' per-stream scratch: built with g++ against a fake of the CUDA calls it makes (no GPU, no CUDA library)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_addresses_handed_out_stay(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / "test_tc_scratch")
    subprocess.run(["g++", "-std=c++17", "-O1", "-x", "c++", "-I", os.path.join(cuda, "include"), os.path.join(ROOT, "tests", "cpp", "test_tc_scratch.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "tc_scratch: ok" in r.stdout, r.stdout
