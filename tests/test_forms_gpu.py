"""The batched form against the plain form on the same uploaded state, bit for
bit: where the two run different kernels (edge EMFs by marching CTAs against
one thread per edge; flux kernels that store more or less), at
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


def _run_both(blocks, coord, W, Bf, steps=2, **kw):
    out = []
    ns = 3 if kw.get("integrator") == fx.INT_ESSPRK10_4 else 2
    for form in (fx.FORM_PLAIN, fx.FORM_BATCHED):
        ctx = fx.Context(Bf is not None, 5.0 / 3.0, coord, **kw)
        ctx.set_mesh(mesh.to_desc(blocks))
        for b in range(len(blocks)):
            w = np.zeros((W.shape[1], ns, W.shape[3]))
            w[:, :2] = W[b]
            f = None
            if Bf is not None:
                f = np.zeros((3, ns, Bf.shape[3]))
                f[:, :2] = Bf[b]
                f = [x.ravel() for x in f]
            ctx.upload_block(b, w.ravel(), f)
        ctx.boundary_fill(1, 0)
        clock = ctx.run(form, steps, 0.4, 1.2, 1.0e30, (0.0, 0.0, 0))
        act = [b for b in range(len(blocks)) if blocks[b].active == 1]
        flux = [ctx.download_array(b, fx.ARR_FLUX, d) for b in (act[0], act[-1]) for d in range(3)]
        out.append((clock, [ctx.download_block(b) for b in act], flux))
        ctx.close()
    assert out[0][0] == out[1][0]
    for (Wa, ea, Ba), (Wb, eb, Bb) in zip(out[0][1], out[1][1]):
        assert np.array_equal(Wa, Wb) and np.array_equal(ea, eb)
        for d in range(3 if Bf is not None else 0):
            assert np.array_equal(Ba[d], Bb[d])
    nv = W.shape[1]
    for n, (a, b) in enumerate(zip(out[0][2], out[1][2])):
        d = n % 3
        core = tuple(slice(2, 19 if q == d else 18) for q in range(3))
        for v in range(6):
            x, y = (f.reshape(20, 20, 5, nv, 4)[:, :, :, v].reshape(20, 20, 20)[core] for f in (a, b))
            assert np.array_equal(x, y)


AMR_COORD = (-0.7, 0.7, -0.7, 0.7, -0.7, 0.7)


@pytest.mark.parametrize("mhd", [True, False])
@pytest.mark.parametrize("use_bj", [False, True])
def test_amr_steps_of_both_forms_are_the_same(mhd, use_bj):
    """Three levels: corrections on the compact fluxes, waves with pairs,
    single operations and face-prolongation groups; steps enough for the
    plain form's graph."""
    blocks = mesh.static_amr_mesh((3,) * 3, AMR_COORD, 2, mesh.ball_refiner((0.1, 0.05, 0.0), (0.4, 0.2)))
    recs = fx.plan_export(fx.make_config(mhd, 5.0 / 3.0, AMR_COORD), mesh.to_desc(blocks), 3) if mhd else None
    W, Bf = problems.amr_blast(blocks, recs, mhd=mhd)
    _run_both(blocks, AMR_COORD, W, Bf, steps=6, use_bj=use_bj)


@pytest.mark.parametrize("root", [(1, 1, 1), (2, 3, 3)])
@pytest.mark.parametrize("recon,integ", [(fx.RECON_MC, fx.INT_RK2), (fx.RECON_WENO3, fx.INT_RK2),
                                         (fx.RECON_MC, fx.INT_ESSPRK10_4)])
@pytest.mark.parametrize("mhd", [True, False])
def test_uniform_steps_of_both_forms_are_the_same(root, recon, integ, mhd):
    blocks = mesh.uniform_mesh(root, COORD)
    W, Bf = problems.fourier_mhd(blocks, nmodes=4, kmax=3)
    if not mhd:
        W, Bf = np.ascontiguousarray(W[:, :6]), None
    _run_both(blocks, COORD, W, Bf, steps=5, recon=recon, integrator=integ)


@pytest.mark.parametrize("mhd", [True, False])
def test_sharded_steps_match_one_device(mhd):
    """Three ranks emulated in one process (flux and EMF records across
    ranks read the compact face arrays) against one context."""
    import threading
    blocks = mesh.static_amr_mesh((3,) * 3, AMR_COORD, 2, mesh.ball_refiner((0.1, 0.05, 0.0), (0.25, 0.1)))
    desc = mesh.to_desc(blocks)
    recs = fx.plan_export(fx.make_config(mhd, 5.0 / 3.0, AMR_COORD), desc, 3) if mhd else None
    W, Bf = problems.amr_blast(blocks, recs, mhd=mhd)

    def field(b):
        return None if Bf is None else [Bf[b, d].ravel() for d in range(3)]

    one = fx.Context(mhd, 5.0 / 3.0, AMR_COORD)
    one.set_mesh(desc)
    for b in range(len(blocks)):
        one.upload_block(b, W[b].ravel(), field(b))
    one.boundary_fill(1, 0)
    clock = one.run(fx.FORM_BATCHED, 2, 0.4, 1.2, 1.0e30, (0.0, 0.0, 0))
    owner = fx.morton_owner(desc, 3)
    group = fx.ShardGroup(3)
    ctxs, got, err = [], [None] * 3, []
    for r in range(3):
        c = fx.Context(mhd, 5.0 / 3.0, AMR_COORD)
        c.shard_set_mesh(desc, owner, 3, r)
        c.attach_group(group)
        for b in np.nonzero(owner == r)[0]:
            c.upload_block(int(b), W[b].ravel(), field(b))
        ctxs.append(c)

    def work(r):
        try:
            ctxs[r].boundary_fill(1, 0)
            got[r] = ctxs[r].run(fx.FORM_BATCHED, 2, 0.4, 1.2, 1.0e30, (0.0, 0.0, 0))
        except Exception as e:  # re-raised below
            err.append(e)
    threads = [threading.Thread(target=work, args=(r,)) for r in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(timeout=300)
    assert not err, err
    assert got == [clock] * 3
    for r in range(3):
        for b in np.nonzero(owner == r)[0]:
            a, c = one.download_block(int(b)), ctxs[r].download_block(int(b))
            assert np.array_equal(a[0], c[0])
            for d in range(3 if mhd else 0):
                assert np.array_equal(a[2][d], c[2][d])
    for c in ctxs + [one]:
        c.close()
    group.close()


def test_driver_loop_stops_and_goes_on_as_the_plain_form():
    """dt carried from step to step (batched RK2) against dt computed per step
    (plain): a run cut short at t_end, a run that starts at t_end, another
    CFL number, and state changed between runs."""
    got = []
    for form in (fx.FORM_PLAIN, fx.FORM_BATCHED):
        ctx, n = _context((2, 2, 4))
        clocks = [ctx.run(form, 3, 0.4, 1.2, 1.0e30, (0.0, 0.0, 0))]
        clocks.append(ctx.run(form, 9, 0.4, 1.2, 1.4 * clocks[0][0], clocks[0]))
        clocks.append(ctx.run(form, 2, 0.4, 1.2, clocks[1][0], clocks[1]))
        clocks.append(ctx.run(form, 2, 0.2, 1.2, 1.0e30, clocks[2]))
        ctx.step(form, 0.5 * clocks[3][1])
        clocks.append(ctx.run(form, 2, 0.2, 2.0, 1.0e30, clocks[3]))
        got.append((clocks, _state(ctx, n)))
        ctx.close()
    assert got[0][0] == got[1][0]
    assert got[0][0][2] == got[0][0][1]
    _same(got[0][1], got[1][1])


@pytest.mark.parametrize("before", [1, 5])
def test_plain_step_inside_a_capture_of_the_callers(before):
    """A plain step that the caller captures on the context's stream, before
    and after the library keeps a graph of its own: launched, it is the step."""
    import torch
    got = []
    for captured in (False, True):
        ctx, n = _context((2, 2, 1))
        dt = 0.3 * ctx.calc_dt(0.4)
        for _ in range(before):
            ctx.step(fx.FORM_PLAIN, dt)
        if captured:
            g = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream())):
                g.capture_begin(capture_error_mode="thread_local")
                ctx.step(fx.FORM_PLAIN, dt, want_dt_src=False)
                g.capture_end()
                g.replay()
                g.replay()
        else:
            for _ in range(2):
                ctx.step(fx.FORM_PLAIN, dt)
        ctx.sync()
        got.append(_state(ctx, n))
        ctx.close()
    _same(got[0], got[1])
