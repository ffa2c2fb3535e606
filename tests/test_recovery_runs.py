"""The row-walking recovery's work list (csrc/knc_runs.h), checked on the host
by tests/cpp/test_runs.cpp."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_runs_cover_every_row_within_one_wave(tmp_path):
    import build as b
    gxx = shutil.which("g++") or shutil.which("c++")
    if gxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "test_runs"
    cuda = Path(b.nvcc()).resolve().parent.parent / "include"
    r = subprocess.run([gxx, "-std=c++17", "-O2", f"-I{b.CSRC}", f"-I{cuda}", "-o", str(exe),
                        str(ROOT / "tests" / "cpp" / "test_runs.cpp")], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
