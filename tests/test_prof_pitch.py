"""Score profiles reach as far as the strips that stage them (no device is touched)."""
import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_profiles_cover_their_strips(tmp_path):
    exe = tmp_path / "prof_pitch"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include",
                    str(ROOT / "tests/cpp/prof_pitch.cpp"), "-o", str(exe)], check=True)
    pairs, short_of = map(int, subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.split())
    assert pairs > 9000 and short_of == 0
