"""Which kernel runs a window (csrc/gf_plan.h), compiled with the host compiler: windows longer than the records
a block stages go to the kernel that reads them from memory."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_window_forms(tmp_path):
    exe = tmp_path / "window_form_test"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "parallelpopgen_b200" / "csrc"),
                    "-I", str(ROOT / "include"), str(ROOT / "tests" / "cpp" / "window_form_test.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip().endswith("OK"), out.stdout
