"""The evaluation's block of small buffers on a fake CUDA runtime (tests/cpp/arena_check.cpp):
a call made inside an evaluation on another device or stream gets memory of its own."""
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_block_serves_its_own_device_and_stream(tmp_path):
    out = tmp_path / "arena_check"
    cmd = ["g++", "-std=c++17", "-O1", "-x", "c++", f"-I{ROOT / 'libuw12_b200' / 'csrc'}",
           "-I/usr/local/cuda/include", str(ROOT / "tests" / "cpp" / "arena_check.cpp"), "-o",
           str(out)]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(out)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
