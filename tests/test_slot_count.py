"""The engine's bound on its mutation count (csrc/gf_plan.h), compiled with the host compiler."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_slot_count(tmp_path):
    exe = tmp_path / "slot_count_test"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "parallelpopgen_b200" / "csrc"),
                    "-I", str(ROOT / "include"), str(ROOT / "tests" / "cpp" / "slot_count_test.cpp"), "-o", str(exe)],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True)
    assert out.returncode == 0 and out.stdout.strip().endswith("OK"), out.stdout
