"""The adjoint's tape keeps more than the one segment every reverse pass needs
only within its limit and half of the memory left after everything else:
tests/cpp/adjoint_tape.cpp."""
import shutil
import subprocess

import pytest

from conftest import ROOT

GIB = 1 << 30
# segments, bytes each, limit, free -> kept
CASES = [
    ((3, GIB, 8 * GIB, 200 * GIB), 3),
    ((63, 3 * GIB, 8 * GIB, 200 * GIB), 2),
    ((6, 3 * GIB // 2, 8 * GIB, 200 * GIB), 5),
    ((4, 9 * GIB, 8 * GIB, 200 * GIB), 1),        # one is over the limit
    ((4, GIB, 8 * GIB, 4 * GIB), 2),              # half of what is free
    ((4, GIB, 8 * GIB, 2 * GIB - 2), 1),
    ((4, GIB, 8 * GIB, 0), 1),
    ((1, 1, 8 * GIB, 200 * GIB), 1),
    ((2000, 0, 8 * GIB, 200 * GIB), 2000),        # no particles
]


def test_kept_segments(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "adjoint_tape")
    subprocess.run(["g++", "-std=c++17", "-O1", "-o", exe, f"{ROOT}/tests/cpp/adjoint_tape.cpp"], check=True)
    lines = "\n".join(" ".join(map(str, c)) for c, _ in CASES)
    r = subprocess.run([exe], input=lines, capture_output=True, text=True, check=True)
    assert [int(v) for v in r.stdout.split()] == [want for _, want in CASES]
