"""The threads that convert a downloaded field: they sleep while its copy is queued
behind other work, and convert every chunk that arrives once."""
import shutil
import subprocess
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent


def test_host_chunks(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = tmp_path / "host_threads"
    subprocess.run([cxx, "-std=c++17", "-O1", "-pthread", "-o", str(exe), str(HERE / "cpu" / "host_threads.cpp")], check=True)
    out = dict(line.split() for line in
               subprocess.run([str(exe)], check=True, capture_output=True, text=True, timeout=120).stdout.splitlines())
    # half a second on one thread that spins would be 0.5
    assert float(out["cpu"]) < 0.1
    assert out["once"] == "1"
