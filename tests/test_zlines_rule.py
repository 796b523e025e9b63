"""The host rule of the whole-line z passes, checked over all forms it accepts (tests/cpp/zlines_rule.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_whole_line_rule(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    exe = str(tmp_path / "zlines_rule")
    cmd = ["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "inq_b200", "csrc"), "-I", os.path.join(cuda, "include"),
           os.path.join(ROOT, "tests", "cpp", "zlines_rule.cpp"), "-o", exe]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
