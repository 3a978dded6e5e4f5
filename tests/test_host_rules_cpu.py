"""Rules of the engine that hold between host threads and between launches,
compiled from the engine's own headers into a program without a device
(tests/cpp/host_rules.cpp)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CXX = shutil.which("g++")


@pytest.mark.skipif(CXX is None, reason="g++ not found")
@pytest.mark.parametrize("rule", ["step", "grid"])
def test_host_rule(tmp_path, rule):
    exe = str(tmp_path / "host_rules")
    r = subprocess.run([CXX, "-std=c++17", "-O1", "-Wall", "-Werror", "-pthread", "-I",
                        os.path.join(ROOT, "apocharmm_b200", "csrc"),
                        os.path.join(ROOT, "tests", "cpp", "host_rules.cpp"), "-o", exe],
                       stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert r.returncode == 0, r.stdout[-3000:]
    r = subprocess.run([exe, rule], stdout=subprocess.PIPE, text=True, timeout=60)
    assert r.returncode == 0, r.stdout
