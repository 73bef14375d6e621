"""The column transforms of the x and y passes, run with host threads as the threads
of a tile: all four kinds, every length, both tile widths, whole and split exchange."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
TOL = {"fp64": 2e-15, "fp32": 1e-6}   # of the largest output; log2(512) stages of half an ulp


def test_column_tiles(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = tmp_path / "columns"
    subprocess.run([cxx, "-std=c++20", "-O1", "-pthread", "-o", str(exe), str(HERE / "cpu" / "columns.cpp")], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=600).stdout
    rows = [line.split() for line in out.splitlines()]
    assert len(rows) == 9 * 3 + 6 * 3   # lengths 8 to 32 have too few lanes for tiles of 4
    for prec, n, pencils, split, err in rows:
        assert float(err) < TOL[prec], (prec, n, pencils, split, err)
