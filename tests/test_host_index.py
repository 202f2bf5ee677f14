"""What the index loader makes of a file's lists (host code alone)."""
import os
import subprocess

from conftest import ROOT


def test_lists_that_no_builder_makes(tmp_path):
    exe = str(tmp_path / "host_index_test")
    src = [os.path.join(ROOT, "tests", "cpp", "host_index_test.cc"),
           os.path.join(ROOT, "genie_gb300", "csrc", "host_index.cc")]
    r = subprocess.run(["g++", "-std=c++17", "-O1"] + src + ["-o", exe, "-lpthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "OK", r.stdout
