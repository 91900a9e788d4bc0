"""The library's device memory where CUDA calls are refused or run out of
memory, on the host against a counting stand-in for the runtime (pool_fake.cpp);
and that no wait's refusal is passed over.
"""
import re
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


def test_every_wait_is_looked_at():
    """A wait that a capture refuses has not waited, and what follows it may free
    what a kernel still uses: no source discards a wait's result."""
    unread = re.compile(r"(^|[;{})]|\bdone:|else)\s*cuda(Device|Stream|Event)Synchronize\s*\([^;]*\)\s*;", re.M)
    for src in sorted(B.CSRC.iterdir()):
        text = re.sub(r"//[^\n]*", "", src.read_text())
        for m in unread.finditer(text):
            line = text[:m.end()].count("\n") + 1
            raise AssertionError(f"{src.name}:{line}: {m.group(0).strip()}")
