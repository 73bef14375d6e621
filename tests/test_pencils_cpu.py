"""The register transforms of the row and column passes, run with host threads
as the lanes of a warp: all four kinds, every row length, both plans."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
TOL = {"fp64": 2e-15, "fp32": 1e-6}   # of the largest output; log2(512) stages of half an ulp


def test_register_transforms(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = tmp_path / "pencils"
    subprocess.run([cxx, "-std=c++20", "-O1", "-pthread", "-o", str(exe), str(HERE / "cpu" / "pencils.cpp")], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=300).stdout
    rows = [line.split() for line in out.splitlines()]
    assert len(rows) == 20
    for prec, n, wide, err in rows:
        assert float(err) < TOL[prec], (prec, n, wide, err)
