"""Handles used from several threads: what the launchers share between them."""
import glob
import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "cpp", "test_once_per_device.cpp")


def test_marks_per_device_under_the_thread_sanitizer(tmp_path):
    def run(source, exe):
        r = subprocess.run(["g++", "-std=c++17", "-O1", "-g", "-fsanitize=thread", source, "-o", exe], capture_output=True, text=True)
        return r if r.returncode else subprocess.run([exe], capture_output=True, text=True, timeout=120)

    plain = tmp_path / "plain.cpp"
    plain.write_text("int main() { return 0; }\n")
    if run(str(plain), str(tmp_path / "plain")).returncode:
        pytest.skip("no thread sanitizer here")
    r = run(SRC, str(tmp_path / "once"))
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr


def test_launchers_keep_no_unguarded_marks():
    """A plain static flag per device, written by whichever handle comes first, is a data race between two handles; the
    memory pool's are read and written under its lock."""
    for path in glob.glob(os.path.join(ROOT, "systemds_b200", "csrc", "*.cu*")):
        found = re.findall(r"\bstatic\s+bool\s+(\w+)\s*\[", open(path).read())
        assert [f for f in found if f != "g_poolTried"] == [], path
