"""The face arrays both forms leave (fluxes, face velocities) whatever the
order in which steps, downloads, per-block entry points and replays of the
caller's own captures come: always those of the last face kernel that ran,
compared bit for bit with the same sequence issued one call at a time."""
import numpy as np
import pytest

import fornaxamr_b200 as fx
from fornaxamr_b200 import mesh, problems

pytestmark = pytest.mark.gpu
COORD = (0.0, 1.0, 0.0, 1.0, 0.0, 1.0)
P, NG, BS = 20, 2, 16


def _initial(root):
    return [np.ascontiguousarray(a) for a in problems.fourier_mhd(mesh.uniform_mesh(root, COORD), nmodes=4, kmax=3)]


def _context(root=(2, 2, 4), mhd=True, **kw):
    blocks = mesh.uniform_mesh(root, COORD)
    W, Bf = _initial(root)
    if not mhd:
        W, Bf = np.ascontiguousarray(W[:, :6]), None
    ctx = fx.Context(mhd, 5.0 / 3.0, COORD, **kw)
    ctx.set_mesh(mesh.to_desc(blocks))
    if ctx.ns == 3:
        W = np.concatenate([W, W[:, :, :1]], 2)
        Bf = None if Bf is None else np.concatenate([Bf, Bf[:, :, :1]], 2)
    ctx.upload_all(np.ascontiguousarray(W), None if Bf is None else np.ascontiguousarray(Bf))
    ctx.boundary_fill(1, 0)
    return ctx, len(blocks)


def _faces(ctx, n):
    """Fluxes [direction][variable, i, j, k] and face velocities of a few blocks."""
    out = []
    for b in sorted({0, n // 2, n - 1}):
        for d in range(3):
            f = ctx.download_array(b, fx.ARR_FLUX, d).reshape(P, P, P // 4, ctx.nv, 4)
            v = ctx.download_array(b, fx.ARR_VRIEMANN, d).reshape(P, P, P // 4, 3, 4)
            out.append((f.transpose(3, 0, 1, 2, 4).reshape(ctx.nv, P, P, P), v.transpose(3, 0, 1, 2, 4).reshape(3, P, P, P)))
    return out


def _same_faces(a, b, variables=None, normal_only=False):
    for n, ((fa, va), (fb, vb)) in enumerate(zip(a, b)):
        assert np.array_equal(fa[:variables], fb[:variables])
        q = slice(n % 3, n % 3 + 1) if normal_only else slice(None)
        assert np.array_equal(va[q], vb[q])


def _state(ctx, n):
    return [ctx.download_block(b) for b in range(n)]


def _same_state(a, b):
    for x, y in zip(a, b):
        assert np.array_equal(x[0], y[0])
        assert len(x[2]) == len(y[2]) and all(np.array_equal(p, q) for p, q in zip(x[2], y[2]))


@pytest.mark.parametrize("nsteps", [1, 3])
def test_a_run_that_takes_no_step_leaves_the_faces(nsteps):
    """Time has reached t_end: the batched run does nothing, to the face
    arrays of the plain step before it as to the state."""
    ctx, n = _context()
    dt = 0.2 * ctx.calc_dt(0.4)
    ctx.step(fx.FORM_BATCHED, dt)
    ctx.step(fx.FORM_PLAIN, dt)
    ctx.flux_update(n - 1, 0, 0)
    ctx.sync()
    want = _faces(ctx, n)
    clock = (1.0, dt, 2)
    assert ctx.run(fx.FORM_BATCHED, nsteps, 0.4, 1.2, 1.0, clock) == clock
    _same_faces(_faces(ctx, n), want)
    ctx.close()


def _capture(ctx, calls):
    import torch
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream())):
        g.capture_begin(capture_error_mode="thread_local")
        calls()
        g.capture_end()
    return g


def _replay(ctx, g):
    import torch
    with torch.cuda.stream(torch.cuda.ExternalStream(ctx.stream())):
        g.replay()
    ctx.sync()


def _update(ctx, n, dt):
    """The per-block entry points on the faces at hand."""
    for b in range(n):
        ctx.mhd_update_emf(b, 0)
        ctx.mhd_update_bf(b, 1, dt)
        ctx._check(ctx.L.fx_update_cells(ctx._h, b, 1, dt, None))


# what the caller captures, with which form of step before the capture and
# between the capture and its replay
@pytest.mark.parametrize("what", ["plain step", "update"])
@pytest.mark.parametrize("before", [fx.FORM_PLAIN, fx.FORM_BATCHED])
@pytest.mark.parametrize("between", [fx.FORM_PLAIN, fx.FORM_BATCHED])
def test_replay_of_a_capture_between_steps_of_either_form(what, before, between):
    got = []
    for captured in (False, True):
        ctx, n = _context()
        dt = 0.2 * ctx.calc_dt(0.4)
        call = {"plain step": lambda: ctx.step(fx.FORM_PLAIN, dt, want_dt_src=False),
                "update": lambda: _update(ctx, n, dt)}[what]
        ctx.step(fx.FORM_BATCHED, dt)  # both forms have left their faces once
        ctx.step(before, dt)
        if captured:
            g = _capture(ctx, call)
            mid = _faces(ctx, n)
        else:
            mid = _faces(ctx, n)
        ctx.step(between, dt)
        if captured:
            _replay(ctx, g)
        else:
            call()
        last = _faces(ctx, n)
        _update(ctx, n, dt)
        ctx.riemann_flux_send()
        ctx.sync()
        got.append((mid, last, _state(ctx, n)))
        ctx.close()
    _same_faces(got[0][0], got[1][0])
    _same_faces(got[0][1], got[1][1])
    _same_state(got[0][2], got[1][2])


@pytest.mark.parametrize("phase,array", [(fx.PHASE_EMF, "ARR_EMF"), (fx.PHASE_CELLS, "ARR_W")])
def test_timed_phases_run_on_the_last_faces(phase, array):
    """A phase timed after a plain step works on that step's face arrays, as
    the per-block entry point does."""
    got = []
    for timed in (True, False):
        ctx, n = _context()
        dt = 0.2 * ctx.calc_dt(0.4)
        ctx.step(fx.FORM_PLAIN, dt)
        if timed:
            ctx.time_phase(phase, 1, dt)
        else:
            for b in range(n):
                if phase == fx.PHASE_EMF:
                    ctx.mhd_update_emf(b, 0)
                else:
                    ctx.update_cells(b, 1, dt)
        ctx.sync()
        got.append([ctx.download_array(b, getattr(fx, array), d) for b in range(n)
                    for d in (range(3) if phase == fx.PHASE_EMF else (0,))])
        ctx.close()
    for a, b in zip(*got):
        assert np.array_equal(a, b)


def _advance(ctx, form, how):
    """Ways to the last face fluxes of a call."""
    dt = 0.2 * ctx.calc_dt(0.4)
    if how == "step":
        ctx.step(form, dt)
        ctx.step(form, dt)
    elif how == "stage":
        ctx.stage(form, 1, dt)
    elif how == "run":
        a = ctx.run(form, 3, 0.1, 1.2, 1.0e30, (0.0, 0.0, 0))
        a = ctx.run(form, 1, 0.1, 1.2, 1.0e30, a)
        ctx.run(form, 2, 0.1, 1.2, 1.0e30, a)
    else:  # the run ends before its steps are used up
        a = ctx.run(form, 9, 0.1, 1.2, 5.0 * dt / 2.0, (0.0, 0.0, 0))
        assert a[0] == 5.0 * dt / 2.0 and a[2] < 9


@pytest.mark.parametrize("mhd,integ,how", [(m, i, h) for m in (True, False) for i, h in
                                           [(fx.INT_RK2, "step"), (fx.INT_RK2, "stage"), (fx.INT_RK2, "run"),
                                            (fx.INT_RK2, "run to t_end"), (fx.INT_ESSPRK10_4, "step"),
                                            (fx.INT_ESSPRK10_4, "run")]])
def test_every_face_of_both_forms_is_the_same(mhd, integ, how):
    """All of a block's faces, the MHD ghost layer of the transverse axes
    among them: six components and the normal velocity of the batched form,
    every component of the plain one; nothing elsewhere."""
    got = []
    for form in (fx.FORM_PLAIN, fx.FORM_BATCHED):
        ctx, n = _context((2, 2, 3), mhd, integrator=integ)
        _advance(ctx, form, how)
        got.append(_faces(ctx, n))
        ctx.close()
    _same_faces(got[0], got[1], variables=6, normal_only=True)
    r = 1 if mhd else 0
    for q, (f, v) in enumerate(got[0]):
        d = q % 3
        m = np.zeros((P, P, P), bool)
        m[tuple(slice(NG, NG + BS + 1) if a == d else slice(NG - r, NG + BS + r) for a in range(3))] = True
        assert (f[0][m] != 0).mean() > 0.99 and (v[d][m] != 0).mean() > 0.99
        assert not f[:, ~m].any() and not v[:, ~m].any()
        if mhd:  # the field flux along the sweep is zero
            assert [bool(c[m].any()) for c in f[6:]] == [c != d for c in range(3)] and all(c[m].any() for c in v)


def test_faces_of_a_run_cut_short_on_three_levels():
    """With coarse/fine corrections of the fluxes: a run that reaches t_end
    early, in both forms."""
    coord = (-0.7, 0.7) * 3
    blocks = mesh.static_amr_mesh((3,) * 3, coord, 2, mesh.ball_refiner((0.1, 0.05, 0.0), (0.4, 0.2)))
    desc = mesh.to_desc(blocks)
    W, Bf = problems.amr_blast(blocks, fx.plan_export(fx.make_config(True, 5.0 / 3.0, coord), desc, 3))
    act = [b for b in range(len(blocks)) if blocks[b].active == 1][::7]
    got = []
    for form in (fx.FORM_PLAIN, fx.FORM_BATCHED):
        ctx = fx.Context(True, 5.0 / 3.0, coord)
        ctx.set_mesh(desc)
        ctx.upload_all(W, Bf)
        ctx.boundary_fill(1, 0)
        dt = ctx.calc_dt(0.2)
        assert ctx.run(form, 9, 0.2, 1.2, 2.5 * dt, (0.0, 0.0, 0))[2] < 9
        got.append([(ctx.download_array(b, fx.ARR_FLUX, d).reshape(P, P, P // 4, 9, 4)[:, :, :, :6],
                     ctx.download_array(b, fx.ARR_VRIEMANN, d).reshape(P, P, P // 4, 3, 4)[:, :, :, d])
                    for b in act for d in range(3)])
        ctx.close()
    for (fa, va), (fb, vb) in zip(*got):
        assert np.array_equal(fa, fb) and np.array_equal(va, vb)


def test_a_batched_step_keeps_what_only_the_plain_form_has():
    """Field fluxes and transverse face velocities of an earlier plain step
    are still there after a batched one, which does not compute them."""
    ctx, n = _context()
    dt = 0.2 * ctx.calc_dt(0.4)
    ctx.step(fx.FORM_PLAIN, dt)
    a = _faces(ctx, n)
    ctx.step(fx.FORM_BATCHED, dt)
    b = _faces(ctx, n)
    ctx.close()
    for q, ((fa, va), (fb, vb)) in enumerate(zip(a, b)):
        assert np.array_equal(fa[6:], fb[6:])
        for c in range(3):
            assert np.array_equal(va[c], vb[c]) == (c != q % 3)


@pytest.mark.parametrize("how", ["autotune", "time_phase"])
def test_timed_face_kernels_leave_every_face(how):
    """As the flux kernel of the plain form leaves them on the same state."""
    ctx, n = _context()
    dt = 0.2 * ctx.calc_dt(0.4)
    for b in range(n):
        ctx.flux_update(b, 0, 0)
    want = _faces(ctx, n)
    ctx.step(fx.FORM_BATCHED, dt)
    ctx.upload_all(*_initial((2, 2, 4)))
    ctx.boundary_fill(1, 0)
    if how == "autotune":
        ctx.autotune()
    else:
        ctx.time_phase(fx.PHASE_FLUX, 2, dt)
    _same_faces(_faces(ctx, n), want, variables=6, normal_only=True)
    ctx.close()
