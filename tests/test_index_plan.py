"""The parallel block index's segments, batches and workspace, on the host
(tests/cpp/index_plan.cpp)."""
from __future__ import annotations

import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_index_plan(tmp_path):
    exe = str(tmp_path / "index_plan")
    subprocess.run(["g++", "-O2", "-std=c++17", "-Wall", "-Werror", "-Wno-unknown-pragmas",
                    "-Wno-maybe-uninitialized", "-I", os.path.join(ROOT, "cuzfp_gb300", "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "cpp", "index_plan.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
