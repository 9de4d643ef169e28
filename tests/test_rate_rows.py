"""The interval-polynomial rows the loader builds (rate columns, angle
fractions) against the reference's interpolation formulas in extended
precision, and their row search at every node, cell edge and neighbouring
double: tests/cpp/rate_rows.cpp, which also derives the allowed error."""
import shutil
import subprocess

import pytest

from conftest import ROOT, TABLES


def test_rows_match_the_interpolation(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "rate_rows")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", exe, f"{ROOT}/tests/cpp/rate_rows.cpp",
                    f"{ROOT}/rrea_feedback_warpx_amrex_geant4_gb300/csrc/host/table_set.cpp", "-lz"], check=True)
    r = subprocess.run([exe, TABLES], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    assert r.stdout.rstrip().endswith("ok")
