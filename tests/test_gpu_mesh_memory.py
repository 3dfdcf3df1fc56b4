"""Chunks meshed together when device memory is short (tests/cpp/mesh_memory_check.cpp, whose own
cudaMalloc refuses what goes past a budget; the GPU's memory is not touched)."""
import subprocess

import pytest

from tests.cpp import build_check

pytestmark = pytest.mark.gpu


def test_smaller_groups_when_memory_is_short(gpu):
    exe = build_check.build("mesh_memory_check")
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "0 failures" in r.stdout
