"""The tickets that the shared-cache attention's key splits meet at: every order of arrival of two calls that overlap
must leave them at zero, or the calls after them would join their splits too early.  Runs on the host, with the code
that the kernel uses."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_overlapping_calls_leave_the_tickets_at_zero(tmp_path):
    exe = tmp_path / "split_ticket_test"
    r = subprocess.run(["/usr/bin/g++", "-std=c++17", "-Wall", "-O1", "-I", os.path.join(ROOT, "litert-lm_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "split_ticket_test.cc"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
