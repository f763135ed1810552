"""Device buffers where memory runs out (tests/cpp/test_alloc.cpp: a fake CUDA on the host)."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parent.parent


def test_alloc_gives_the_pool_back_and_tries_again(tmp_path):
    exe = tmp_path / "test_alloc"
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", "/usr/local/cuda/include",
                        str(ROOT / "tests" / "cpp" / "test_alloc.cpp"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "ALL PASSED" in r.stdout, r.stdout + r.stderr
