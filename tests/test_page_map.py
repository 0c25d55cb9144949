"""How many pages of a cache the attention on tcgen05 reaches.  Runs on the host, with the code that makes its tensor maps."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_every_page_within_32_tb_is_counted(tmp_path):
    exe = tmp_path / "page_map_test"
    r = subprocess.run(["/usr/bin/g++", "-std=c++17", "-Wall", "-O1", "-I", os.path.join(ROOT, "litert-lm_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "page_map_test.cc"), "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
