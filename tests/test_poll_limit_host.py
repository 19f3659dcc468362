"""How long the scanner blocks of the digit pass and of unique wait for their first count and for a
later one (tests/cpp/poll_limit_test.cpp runs the device code's rule against a clock of its own).  No
GPU: a wait of this kind is not made to run out on one."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_a_scanner_outlasts_a_kernel_that_holds_the_other_sms(tmp_path):
    exe = str(tmp_path / "poll_limit_test")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-I", os.path.join(ROOT, "ilgpu_b200", "csrc"),
                           os.path.join(HERE, "cpp", "poll_limit_test.cpp"), "-o", exe])
    run = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stdout + run.stderr


def test_the_scanners_use_it():
    """Neither scanner counts its polls by itself."""
    for name, function in (("digit_pass.cuh", "scan_counts"), ("unique.cu", "scan_tile_counts")):
        text = open(os.path.join(ROOT, "ilgpu_b200", "csrc", name)).read()
        body = text[text.index(f" {function}("):]
        body = body[:body.index("\n}\n")]
        assert "ScannerPolls" in body and "kMaxSpin" not in body, name
