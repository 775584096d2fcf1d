"""Builds and runs tests/cpp/test_device_mem.cpp: buffers whose growth fails (no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_buffers_survive_a_failed_allocation(tmp_path):
    exe = str(tmp_path / "test_device_mem")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "test_device_mem.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "0 failed" in r.stdout, r.stdout + r.stderr
