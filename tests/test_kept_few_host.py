"""How many on-chip plans a batch keeps (tests/cpp/kept_few_check.cpp): the last few, however many
settings a tuner goes through. No GPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_the_last_few_are_kept(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "kept_few_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "planet_game_gb300" / "csrc"),
                    str(ROOT / "tests" / "cpp" / "kept_few_check.cpp"), "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr
