"""What a process finds out or sets once a device (kernel attributes, the limits that follow from
them), checked on the host (tests/cpp/per_device_check.cpp), and that no kernel attribute is set
once a process: a function attribute holds on one device, so a second device's launches of a
cluster or of more than 48 KB of shared memory would be refused. No GPU."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "planet_game_gb300" / "csrc"


def test_values_are_kept_per_device(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "per_device_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", str(CSRC),
                    str(ROOT / "tests" / "cpp" / "per_device_check.cpp"), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr


def test_no_kernel_attribute_is_set_once_a_process():
    sources = [f for pattern in ("*.cu", "*.cuh", "*.cpp", "*.hpp") for f in CSRC.rglob(pattern)]
    users = [f for f in sources if "cudaFuncSetAttribute(" in f.read_text()]
    assert users
    # a static initialiser (`static const bool ready = [] { ... }();`) that sets one
    once = re.compile(r"static const [^;{]*= \[\] ?\{((?!\n    \}\(\);).)*cudaFuncSetAttribute\(", re.S)
    assert [f.name for f in users if once.search(f.read_text())] == []
