"""The barrier at which the threads of a block learn that a bounded wait gave up: whoever saw it when, all take the same
branch.  Runs on the host, with the code that the kernels use."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_threads_leave_together(tmp_path):
    exe = tmp_path / "block_vote_test"
    r = subprocess.run(["/usr/bin/g++", "-std=c++17", "-Wall", "-O1", "-pthread", "-I", os.path.join(ROOT, "litert-lm_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "block_vote_test.cc"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
