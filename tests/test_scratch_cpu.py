"""The growth rule of a stream's scratch, against a fake driver: a block whose address a captured graph holds outlives every growth."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_scratch_growth_rule(tmp_path):
    exe = tmp_path / "scratch_selftest"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", f"-I{ROOT / 'halo_b200' / 'csrc'}",
                    str(ROOT / "tests" / "native" / "scratch_selftest.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
