"""Rounding error of the reverse sweep's face, 64-bit against 80-bit
(tests/adjoint_error_check.cpp), over 200000 seeded faces."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_face_adjoints_lose_nothing_to_the_shared_divisions(tmp_path):
    """Mean relative error 3.417e-16; with every product divided by itself, as
    before adjoints shared a division, 3.457e-16 on the same faces.  The
    arithmetic is IEEE double on both sides, so the figure does not move."""
    exe = str(tmp_path / "adjoint_error_check")
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-fno-fast-math", "-std=c++17",
                    "-I" + os.path.join(ROOT, "fornaxamr_b200", "csrc"),
                    os.path.join(HERE, "adjoint_error_check.cpp"), "-o", exe], check=True, capture_output=True, timeout=300)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=300).stdout
    used, mean = re.match(r"(\d+) of 200000 faces, mean (\S+),", out).groups()
    assert int(used) > 199000, out
    assert float(mean) < 3.44e-16, out
