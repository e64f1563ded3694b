"""The tiles' device point numbers, checked on the host: compiles
tests/tile_numbers_check.cu (host code only) with the library's own flags and
runs it."""

from __future__ import annotations

import subprocess
import sys
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]


def run_host_check(name, tmp_path):
    sys.path.insert(0, str(REPO / "in-house-sem_b200"))
    try:
        import build
    finally:
        sys.path.pop(0)
    try:
        nvcc = build.nvcc()
    except RuntimeError:
        pytest.skip("nvcc not available")
    exe = tmp_path / name
    cmd = [nvcc, *build.NVCC_FLAGS, "-I", str(build.CSRC), str(REPO / "tests" / f"{name}.cu"), "-o", str(exe)]
    res = subprocess.run(cmd, capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-3000:]
    run = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0 and run.stdout.startswith("ok"), run.stdout + run.stderr


def test_device_point_numbers(tmp_path):
    run_host_check("tile_numbers_check", tmp_path)
