"""The batched form against the plain form on the same uploaded state, bit for
bit: where the two run different kernels (edge EMFs by marching CTAs against
one thread per edge; compact face arrays against the reference's tiles), at
block counts on both sides of each launch rule."""
import numpy as np
import pytest

import fornaxamr_b200 as fx
from fornaxamr_b200 import mesh, problems

pytestmark = pytest.mark.gpu
COORD = (0.0, 1.0, 0.0, 1.0, 0.0, 1.0)


def _context(root, eta=0.0, rho_scale=1.0, seeds=(1, 2, 3), **kw):
    blocks = mesh.uniform_mesh(root, COORD)
    W, Bf = problems.fourier_mhd(blocks, nmodes=4, kmax=3, seeds=seeds)
    if rho_scale != 1.0:
        # same pressure and field, density about the artificial-resistivity floor
        W[:, 0] *= rho_scale
        W[:, 4] /= rho_scale
        W[:, 5] = 0.2 + 0.1 * (W[:, 0] / rho_scale - 0.7)
    ctx = fx.Context(True, 5.0 / 3.0, COORD, mhd_eta=eta, **kw)
    ctx.set_mesh(mesh.to_desc(blocks))
    ctx.upload_all(np.ascontiguousarray(W), np.ascontiguousarray(Bf))
    ctx.boundary_fill(1, 0)
    return ctx, len(blocks)


def _state(ctx, n):
    return [ctx.download_block(b) for b in range(n)]


def _same(a, b):
    for (Wa, ea, Ba), (Wb, eb, Bb) in zip(a, b):
        assert np.array_equal(Wa, Wb) and np.array_equal(ea, eb)
        for d in range(3):
            assert np.array_equal(Ba[d], Bb[d])


# 15 / 16 blocks: one thread per edge / marching CTAs; 16 and 34 blocks: 17
# chunks, 36: 17 by the division, 75: 8 chunks, 297: 2 chunks
@pytest.mark.parametrize("root", [(1, 3, 5), (2, 2, 4), (2, 17, 1), (3, 3, 4), (3, 5, 5), (3, 9, 11)])
@pytest.mark.parametrize("eta,rho", [(0.0, 1.0), (1e-3, 1.0), (0.0, 1.0e13)])
def test_stage_of_both_forms_is_the_same(root, eta, rho):
    if rho > 1 and len(mesh.uniform_mesh(root, COORD)) > 100:
        pytest.skip("the dense case needs no second large mesh")
    out = []
    for form in (fx.FORM_PLAIN, fx.FORM_BATCHED):
        ctx, n = _context(root, eta, rho)
        # the artificial eta (about 1e11) diffuses a cell in 1e-15
        dt = 0.2 * ctx.calc_dt(0.4) if rho == 1 else 1e-17
        ctx.stage(form, 1, dt)
        ctx.stage(form, 2, dt)
        emf = [ctx.download_array(b, fx.ARR_EMF, d) for b in (0, n // 2, n - 1) for d in range(3)]
        out.append((_state(ctx, n), emf))
        ctx.close()
    _same(out[0][0], out[1][0])
    for a, b in zip(out[0][1], out[1][1]):
        assert np.array_equal(a, b)


def test_plain_entry_points_after_a_batched_step():
    """The face arrays a batched step leaves serve the plain entry points and
    the downloads: cells updated again from them give the plain form's state."""
    got = []
    for form in (fx.FORM_PLAIN, fx.FORM_BATCHED):
        ctx, n = _context((2, 2, 4), gravity=True)
        dt = 0.2 * ctx.calc_dt(0.4)
        ctx.step(form, dt)
        vr = [ctx.download_array(b, fx.ARR_VRIEMANN, d).reshape(400, 5, 3, 4)[:, :, d] for b in (0, n - 1)
              for d in range(3)]
        ctx.step(form, dt)
        for b in range(n):
            ctx.mhd_update_emf(b, 0)
            ctx.mhd_update_bf(b, 1, dt)
            ctx.update_cells(b, 1, dt)
        got.append((_state(ctx, n), vr))
        ctx.close()
    _same(got[0][0], got[1][0])
    for d in range(3):
        m = np.zeros((20, 20, 20), bool)
        m[tuple(slice(2, 19 if q == d else 18) for q in range(3))] = True
        for q in (0, 1):
            a, b = (g[1][3 * q + d].reshape(20, 20, 20) for g in got)
            assert np.array_equal(a[m], b[m])
