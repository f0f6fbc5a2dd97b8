"""The adjoint of the ghost fill clears what the fill writes, from the lists
that the fill itself runs (pairs and single copies); its own tables are the
gathers alone."""
import numpy as np
import pytest

import fornaxamr_b200 as fx
from fornaxamr_b200 import mesh, problems

pytestmark = pytest.mark.gpu
COORD = (0.0, 1.0, 0.0, 1.0, 0.0, 1.0)
P, NG = 20, 2
NFACE = P * P * (P + 1)


def _program(root, which):
    desc = mesh.to_desc(mesh.uniform_mesh(root, COORD))
    return fx.plan_export(fx.make_config(True, 5.0 / 3.0, COORD), desc, which)


def _context(root):
    blocks = mesh.uniform_mesh(root, COORD)
    W, Bf = problems.fourier_mhd(blocks, nmodes=4, kmax=2)
    ctx = fx.Context(True, 5.0 / 3.0, COORD)
    ctx.set_mesh(mesh.to_desc(blocks))
    ctx.upload_all(W, Bf)
    ctx.boundary_fill(1, 0)
    return ctx, len(blocks), W.size


@pytest.mark.parametrize("root", [(1, 1, 1), (2, 3, 1), (3, 3, 3)])
def test_ghosts_carry_no_adjoint_past_the_initial_fill(root):
    """What the fill wrote has no sensitivity left; every ghost cell is such,
    and nearly every ghost face."""
    ctx, nb, n = _context(root)
    ctx.adjoint_forward(2, 0.1 * ctx.calc_dt(0.4))
    # seeds everywhere, ghost cells and faces and both stage slots among them
    rng = np.random.default_rng(7)
    Wb, Bb = ctx.adjoint_backward(rng.standard_normal(n), rng.standard_normal(nb * 6 * NFACE), initial_fill=True)
    ctx.close()
    a = slice(NG, P - NG)
    ghost = np.ones((P, P, P), bool)
    ghost[a, a, a] = False
    Wb = Wb.reshape(nb, 9, 2, P, P, P)[:, :, 0]
    assert np.isfinite(Wb).all() and Wb[:, :, a, a, a].any()
    assert not Wb[:, :, ghost].any()
    face = _program(root, 1)[0]
    dst = np.zeros((nb, 3, NFACE), bool)
    dst[face[:, 0] >> 15, face[:, 2] & 3, face[:, 0] & 32767] = True
    assert dst.mean() > 0.4
    Bb = Bb.reshape(nb, 3, 2, NFACE)[:, :, 0]
    assert np.isfinite(Bb).all() and Bb.any() and not Bb[dst].any()


def test_first_gradient_uploads_no_second_copy_of_the_program():
    """Device memory of a first gradient: states, adjoints and the gathers
    (8 bytes per read, 16 per element read), not the operations again (16
    bytes per copy, 32 per cell of the field)."""
    import torch
    root = (4, 4, 4)
    ctx, nb, n = _context(root)
    nf = nb * 6 * NFACE
    (cell, w), (face, _), (field, _) = (_program(root, k) for k in (0, 1, 4))
    assert len(w) == 2  # one wave
    keys = [face[:, 1].astype(np.int64) * 4 + (face[:, 2] & 3)]
    keys += [field[:, 1 + q].astype(np.int64) * 4 + q // 2 for q in range(6)]
    sources = len(np.unique(cell[:, 1])) + len(np.unique(np.concatenate(keys)))
    dt = 0.1 * ctx.calc_dt(0.4)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    ctx.adjoint_forward(1, dt)
    torch.cuda.synchronize()
    used = free - torch.cuda.mem_get_info()[0]
    ctx.close()
    states = 8 * (3 * (n + nf) + 2 * nb * 3 * P ** 3)
    gathers = 8 * (len(cell) + len(face) + 6 * len(field)) + 16 * sources
    tables = 16 * (len(cell) + len(face)) + 32 * len(field)
    grain = 6 * (2 << 20)  # an allocation is a multiple of 2 MB
    assert tables > 1.5 * grain
    assert used < states + gathers + grain
