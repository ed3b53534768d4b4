"""The packed tables of the fast and scores builds, walked on the host as the
kernels walk them.  The firing pass takes channels in blocks of four, so the
tables hold every channel of the last block: those past the model's have no
entries, and a draw that marks one of them writes nowhere."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_every_channel_of_the_last_block_has_its_entries_and_no_others(tmp_path):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no g++")
    lib = ROOT / "tau_leaping_gb300"
    exe = tmp_path / "check"
    r = subprocess.run([gxx, "-std=c++17", "-I", str(lib / "csrc"), str(ROOT / "tests" / "fast_tables_check.cpp"),
                        "-L", str(lib), "-ltl", f"-Wl,-rpath,{lib}", "-o", str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
