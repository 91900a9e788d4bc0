"""The library's device memory where CUDA calls are refused or run out of
memory, on the host against a counting stand-in for the runtime (pool_fake.cpp).
"""
import subprocess
from pathlib import Path

from ascent_gb300 import build as B

HERE = Path(__file__).resolve().parent


def test_refused_calls(tmp_path):
    exe = tmp_path / "pool_fake"
    cuda = Path(B._nvcc()).resolve().parents[1] / "include"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(cuda), str(HERE / "pool_fake.cpp"),
                    str(B.CSRC / "gvr_pool.cpp"), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout
