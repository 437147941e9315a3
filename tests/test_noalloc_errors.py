"""bhr_step_noalloc on its error paths, with the CUDA runtime and the launches
replaced by fakes that can fail (noalloc_fake.cpp)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_what_failed_calls_leave_behind(tmp_path):
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    csrc = os.path.join(ROOT, "bh_ringdown_b200", "csrc")
    exe = str(tmp_path / "noalloc_fake")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I", os.path.join(ROOT, "include"), "-I", csrc, "-I",
                    os.path.join(cuda, "include"), "-o", exe, os.path.join(ROOT, "tests", "noalloc_fake.cpp"),
                    "-x", "c++", os.path.join(csrc, "bhr_noalloc.cu")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
