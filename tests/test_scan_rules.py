"""Builds and runs tests/cpp/test_scan_rules.cpp: which scan an IVFPQ search takes (no GPU)."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_rules_of_the_ivfpq_scans(tmp_path):
    exe = str(tmp_path / "test_scan_rules")
    subprocess.run(["/usr/bin/g++", "-std=c++17", "-O1", "-I", "/usr/local/cuda/include",
                    os.path.join(ROOT, "tests", "cpp", "test_scan_rules.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and "0 failed" in r.stdout, r.stdout + r.stderr
