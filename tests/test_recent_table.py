"""The table that keeps a handle's tensor maps: with more arrays than places (long
segments of the adjoint) the ones in use stay and the others make room."""
import os
import subprocess

from conftest import ROOT


def test_more_keys_than_places(tmp_path):
    exe = tmp_path / "table"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", os.path.join(ROOT, "openpfc_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_recent_table.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0, p.stdout
