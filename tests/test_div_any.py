"""The frontend quantiser reconstructs its Y coefficients with a division by the
block's scale through its rounded reciprocal and two corrections (`div2_any` in
cujpegxl_b200/csrc/frontend.cu). Checked against the IEEE division on the host,
whose single arithmetic and FMA round as the GPU's."""

from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

REPO = Path(__file__).resolve().parents[1]


@pytest.mark.skipif(shutil.which("gcc") is None, reason="needs gcc")
def test_division_by_any_scale_is_ieee(tmp_path):
    exe = tmp_path / "div_any_check"
    subprocess.run(["gcc", "-O2", "-march=native", "-ffp-contract=off",
                    str(REPO / "tests" / "cpu_checks" / "div_any_check.c"), "-o", str(exe), "-lm"],
                   check=True, capture_output=True, text=True, timeout=300)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert ", 0 mismatching" in r.stdout
