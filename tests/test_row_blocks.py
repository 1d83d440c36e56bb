"""Unaligned rows are read as the 16-byte blocks that cover them, except where
one would leave the frame (csrc/row_blocks.h): the rule, compiled as a host
program, against every byte that the block loads read."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "openpiv-cxx_gb300", "csrc")


def test_blocks_stay_in_the_frame(tmp_path):
    exe = tmp_path / "test_row_blocks"
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", CSRC,
                    os.path.join(HERE, "cpp", "test_row_blocks.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("ok")
