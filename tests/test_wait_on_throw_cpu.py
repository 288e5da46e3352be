"""A call that fails waits for its copies: the guard that the GPU paths hold, on the
CPU against a counting stand-in for the CUDA call."""
import os
import subprocess

from faz_gb300 import build as B

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_scopes_left_by_exceptions_wait(tmp_path):
    exe = str(tmp_path / "wait_on_throw_check")
    subprocess.check_call(["g++", "-O1", "-std=c++17", "-I" + B.cuda_include(), "-o", exe,
                           os.path.join(ROOT, "tests", "wait_on_throw_check.cpp"), "-lpthread"])
    r = subprocess.run([exe], stdout=subprocess.PIPE, text=True)
    assert r.returncode == 0, r.stdout
