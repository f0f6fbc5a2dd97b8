"""The ghost fill's operations as packed for the device (neighbouring copies
joined to pairs) are the compiled program's, wave by wave and in order, and most
are joined: built with the host compiler from fornaxamr_b200/csrc/fx_plan.cpp (tests/plan_pack_check.cpp)."""
import os
import shutil
import subprocess

import pytest

import fornaxamr_b200 as fx
from fornaxamr_b200 import mesh

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA_INC = "/usr/local/cuda/include"


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(CUDA_INC), reason="needs g++ and the CUDA headers")
def test_packed_program_holds_the_same_operations(tmp_path):
    exe = str(tmp_path / "plan_pack_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-pthread", f"-DFX_NG={fx.NG}", "-I" + CUDA_INC,
                    "-I" + os.path.join(ROOT, "fornaxamr_b200", "csrc"), os.path.join(HERE, "plan_pack_check.cpp"),
                    os.path.join(ROOT, "fornaxamr_b200", "csrc", "fx_plan.cpp"), "-o", exe],
                   check=True, capture_output=True, timeout=600)
    c = (-0.7, 0.7, -0.7, 0.7, -0.7, 0.7)
    meshes = {
        "one": (mesh.uniform_mesh((1, 1, 1), c), True, (0,) * 6),
        "uniform": (mesh.uniform_mesh((3, 2, 4), c), True, (0,) * 6),
        "amr": (mesh.static_amr_mesh((2,) * 3, c, 2, mesh.ball_refiner((0.1, 0.05, 0.0), (0.4, 0.2))), True, (0,) * 6),
        "hydro": (mesh.uniform_mesh((5, 1, 2), c), False, (1, 1, 2, 2, 3, 0)),
    }
    names, joined = [], []
    for name, (blocks, mhd, bc) in meshes.items():
        prefix = str(tmp_path / name)
        with open(prefix + ".cfg", "wb") as f:
            f.write(bytes(fx.make_config(mhd, 5.0 / 3.0, c, bc)))
        with open(prefix + ".desc", "wb") as f:
            f.write(bytes(mesh.to_desc(blocks)))
        (joined if name in ("uniform", "amr") else names).append(prefix)
    r = subprocess.run([exe] + names + ["--"] + joined, capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    print(r.stdout)
