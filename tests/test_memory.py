"""The plans' device memory (csrc/dcpse_memory.h) over a fake runtime, on the
host: reuse only after a wait, waits by cudaFree alone, refusals, threads."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_device_memory_over_a_fake_runtime(tmp_path):
    exe = str(tmp_path / "memory")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", os.path.join(ROOT, "tests", "cpp", "test_memory.cpp"),
                    "-o", exe, "-I" + os.path.join(ROOT, "openfpm_numerics_gb300", "csrc")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
