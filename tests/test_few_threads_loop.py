"""The chunked host-thread loop where the host gives few threads or none
(efs_host.h) on the CPU: tests/host/few_threads_loop_test.cpp compiled with g++
against the header libefs.so includes."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT


@pytest.mark.skipif(shutil.which("g++") is None, reason="no g++")
def test_loop_with_few_threads(tmp_path):
    exe = tmp_path / "few_threads_loop_test"
    src = os.path.join(ROOT, "tests", "host", "few_threads_loop_test.cpp")
    inc = os.path.join(ROOT, "efs_b200", "csrc")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", "-I", inc, "-o", str(exe), src], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
