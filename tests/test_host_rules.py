"""Rules that the library's host side decides by, compiled and run without a GPU."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.parametrize("name", ["test_pq_shape"])
def test_host_rules(tmp_path, name):
    exe = os.path.join(str(tmp_path), name)
    subprocess.check_call(["/usr/bin/g++", "-std=c++17", "-O1", "-Wall", "-o", exe, os.path.join(ROOT, "tests", "cpp", name + ".cpp")])
    res = subprocess.run([exe], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, timeout=60)
    assert res.returncode == 0, res.stdout.decode()
