"""The counters that the second launch of a pass leaves for the next one
(csrc/flag_counters.h), compiled as a host program, through every order of the
CTAs' updates, of launches that overlap too."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "openpiv-cxx_gb300", "csrc")


def test_counters_end_at_zero(tmp_path):
    exe = tmp_path / "test_flag_counters"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", CSRC,
                    os.path.join(HERE, "cpp", "test_flag_counters.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok")
