"""The far-field pass's local expansion, compiled for the host: its leading
sums are compensated, quadrupoles included."""
from __future__ import annotations

import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_leading_sums_are_compensated(tmp_path):
    exe = tmp_path / "localexp_test"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I",
                    str(ROOT / "petar_gb300" / "csrc" / "gpuforce"), "-x", "c++",
                    str(ROOT / "tests" / "cpp" / "localexp_test.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
