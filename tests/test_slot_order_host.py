"""What puts a tile of the radix sort, or the words of the sort in one block and of the partition into buckets, in
order when a warp's atomics were not served in lane order, and the check that finds such a tile
(tests/cpp/slot_order_test.cpp runs the kernels' own code on threads of the host, on slots that are out of order).
No GPU."""
import os
import subprocess

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_tiles_that_came_out_of_order(tmp_path):
    exe = str(tmp_path / "slot_order_test")
    subprocess.check_call(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "ilgpu_b200", "csrc"),
                           os.path.join(HERE, "cpp", "slot_order_test.cpp"), "-o", exe])
    run = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stdout + run.stderr
