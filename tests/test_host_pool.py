"""Host thread pool of the plan-time table builders."""

from __future__ import annotations

import os
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_every_item_once_and_exceptions_reach_the_caller(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "host_pool_check")
    subprocess.run([cxx, "-std=c++20", "-O1", "-pthread", "-I", os.path.join(ROOT, "loki_b200", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "cpp", "host_pool_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", (r.returncode, r.stdout, r.stderr)
