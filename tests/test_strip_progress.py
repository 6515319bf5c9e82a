"""Progress words of chained bit-plane strips, for sequences of more strips than 16
bits count (no device is touched)."""
import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_progress_words_grow_over_all_strips(tmp_path):
    exe = tmp_path / "strip_progress"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.environ.get("CUDA_HOME", "/usr/local/cuda") + "/include", str(ROOT / "tests/cpp/strip_progress.cpp"),
                    "-o", str(exe), "-L", str(ROOT / "msa_b200"), "-lmsa_b200", f"-Wl,-rpath,{ROOT / 'msa_b200'}"],
                   check=True)
    strips, columns, wrong = map(int, subprocess.run([str(exe)], capture_output=True, text=True, timeout=60, check=True)
                                 .stdout.split())
    assert strips > 65536 and columns == 150   # the job is chained on bit planes
    assert wrong == 0
