"""From which sizes on stages walk the tiles back and forth (turning_rule.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_sizes_from_which_stages_turn(tmp_path):
    exe = str(tmp_path / "turning_rule")
    subprocess.run(["g++", "-std=c++17", "-w", "-I", os.path.join(ROOT, "include"), "-I",
                    os.path.join(ROOT, "bh_ringdown_b200", "csrc"), "-I",
                    os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "include"), "-o", exe,
                    os.path.join(ROOT, "tests", "turning_rule.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
