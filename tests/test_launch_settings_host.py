"""The launch shapes that a batch's settings report are the ones its launches take, at level sizes
on both sides of every default's line (tests/cpp/launch_settings_check.cpp, linked with the
library). No GPU; that the shapes never change a result is tests/test_autotune_gpu.py's."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_launch_shapes_are_the_ones_set(tmp_path):
    from planet_game_gb300 import build, capi

    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "launch_settings_check"
    cuda = build.CUDA_HOME
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(build.CSRC), "-I", str(cuda / "include"),
                    str(ROOT / "tests" / "cpp" / "launch_settings_check.cpp"), str(capi.LIBRARY), "-L", str(cuda / "lib64"),
                    "-lcudart", f"-Wl,-rpath,{capi.LIBRARY.parent}:{cuda / 'lib64'}", "-o", str(exe)], check=True,
                   capture_output=True, text=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0 and out.stdout.strip() == "OK", out.stdout + out.stderr
