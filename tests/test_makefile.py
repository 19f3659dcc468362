"""The libraries build without Python and without torch, which only the host path of the Python mirror
needs (what make would run; nothing is compiled)."""
import os
import subprocess
import sys

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ilgpu_b200", "csrc")


def _make(python, *targets):
    return subprocess.run(["make", "-n", "-B", "-C", CSRC, "PYTHON=" + python, *targets], capture_output=True, text=True)


def test_without_torch(tmp_path):
    bare = tmp_path / "python"   # a Python that does not find torch
    bare.write_text(f'#!/bin/sh\nexec {sys.executable} -S -I "$@"\n')
    bare.chmod(0o755)
    for python in (str(bare), str(tmp_path / "no-python")):
        run = _make(python)
        assert run.returncode == 0 and not run.stderr, run.stderr
        assert "libb200alg.so" in run.stdout and "libb200alg_mg.so" in run.stdout and "host_calls.cpp" not in run.stdout
    assert subprocess.run(["make", "-B", "-C", CSRC, "PYTHON=" + str(bare), "host"], capture_output=True).returncode != 0


def test_with_torch():
    run = _make(sys.executable)
    assert run.returncode == 0 and "libb200alg.so" in run.stdout and "host_calls.cpp" in run.stdout, run.stderr
