"""State that the kernel layer keeps per device: compiled from its header and run on the host."""
import os
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent


def test_once_per_device(tmp_path):
    gxx = shutil.which("g++")
    if not gxx:
        pytest.skip("g++ not available")
    exe = tmp_path / "per_device"
    res = subprocess.run([gxx, "-std=c++17", "-O1", str(ROOT / "tests/native/per_device.cc"), "-o", str(exe), "-lpthread"], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr[-4000:]
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60, env=dict(os.environ))
    assert res.returncode == 0, res.stdout + res.stderr


def test_kernel_attributes_are_not_set_once_per_process():
    """A limit of shared memory belongs to the device that is current when it is set."""
    for src in sorted((ROOT / "csrc").rglob("*.cu")):
        assert not re.search(r"static\s+(const\s+)?cudaError_t\s+\w+\s*=", src.read_text()), f"{src.name}: an attribute set on the first device only"
