"""The face kernel's solver compiled for the host (tests/face_solver_check.cpp)
against the plain-C restatement (oracle/fx_oracle.c), bit for bit: halved MC
slope, one-sided WENO values, HLLD (cheap checks and the checks themselves, one
side's energy and composition), HLLC.  No tolerance: the
same IEEE operations on selected operands."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_host_build_of_the_face_solver_matches_the_restatement(tmp_path):
    exe = str(tmp_path / "face_solver_check")
    flags = ["-O2", "-ffp-contract=off", "-fno-fast-math"]
    subprocess.run(["gcc", *flags, "-c", os.path.join(ROOT, "oracle", "fx_oracle.c"), "-o", str(tmp_path / "o.o")],
                   check=True, timeout=300)
    subprocess.run(["g++", *flags, "-std=c++17", "-I" + os.path.join(ROOT, "fornaxamr_b200", "csrc"),
                    os.path.join(HERE, "face_solver_check.cpp"), str(tmp_path / "o.o"), "-lm", "-o", exe],
                   check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
