"""Shared memory limits are raised per handle: no kernel's limit hangs on a flag
of the process, which a second device (or a second thread) would share."""
import glob
import os
import re
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "fem_b200", "csrc")


def test_once_per_handle(tmp_path):
    exe = str(tmp_path / "smem_limits")
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "test_smem_limits.cpp")], check=True)
    assert subprocess.run([exe], capture_output=True, text=True).stdout.strip() == "ok"


def test_every_limit_goes_through_the_handle():
    calls = {}
    for path in glob.glob(os.path.join(CSRC, "*")):
        with open(path) as f:
            src = re.sub(r"//[^\n]*", "", f.read())
        assert not re.search(r"static\s+bool", src), path
        n = src.count("cudaFuncSetAttribute(")
        if n:
            calls[os.path.basename(path)] = n
    assert calls == {"state.cuh": 1}   # allow_smem
