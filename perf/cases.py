"""The work a user of this framework has it do, as measurable cases.

A case is one stretch of a user's run between two outputs: the device holds
the mesh and the state, `run` advances it by some driver steps through the
public entry points (`Context.run`, the adjoint pair) and reads the active
region of the new state back into page-locked host arrays, as a program does
that writes a dump or hands the state to its own analysis.  The state goes on
from pass to pass, like a simulation.

Kinds:
  uniform   single-level mesh of nx x ny x nz blocks of 16^3 cells, MHD (HLLD,
            constrained transport) or hydro (HLLC), MC or WENO-Z3
            reconstruction, RK2 or eSSPRK10_4, batched or plain form
  mirror    the drop-in's default mode: every step uploads the state, steps
            and downloads it
  blast     static AMR, magnetised blast, three levels
  collapse  static AMR with a gravity array, four levels
  adjoint   N stored steps forward, then the reverse sweep (a gradient)

Sizes come from bench.py, the workload module and the tests: 8 to 512 blocks.
Inputs are seeded sums of Fourier modes (density, pressure, velocity, vector
potential), the amplitudes of the benchmark's initial state.
"""
from __future__ import annotations

import functools
import math
import random

import numpy as np
import torch

import fornaxamr_b200 as fx
from fornaxamr_b200 import mesh

BS, NG = 16, 2
P = BS + 2 * NG
CFL, DT_FACTOR, T_END = 0.4, 1.2, 1.0e30
F8 = torch.float64


def listed():
    u = dict(kind="uniform", mhd=True, recon="mc", integrator="rk2", form="batched")
    return [
        # a small box or a test problem: launches and latency count
        dict(u, name="mhd_2x2x2", nx=2, ny=2, nz=2, steps=32),
        # an ordinary run on an uneven box
        dict(u, name="mhd_3x5x7", nx=3, ny=5, nz=7, steps=16),
        # the headline benchmark's mesh, 128^3
        dict(u, name="mhd_8x8x8", nx=8, ny=8, nz=8, steps=32),
        # the higher-order reconstruction
        dict(u, name="mhd_weno3_6x6x6", nx=6, ny=6, nz=6, steps=8, recon="weno3"),
        # the ten-stage integrator
        dict(u, name="mhd_ess_4x4x4", nx=4, ny=4, nz=4, steps=4, integrator="ess"),
        # a shock-tube shaped hydro run: one block thick
        dict(u, name="hydro_64x1x1", nx=64, ny=1, nz=1, steps=32, mhd=False),
        # an ordinary hydro box
        dict(u, name="hydro_6x6x6", nx=6, ny=6, nz=6, steps=16, mhd=False),
        # the block-by-block drop-in form
        dict(u, name="plain_3x3x3", nx=3, ny=3, nz=3, steps=2, form="plain"),
        # the drop-in binding's mirror mode: the host owns the state
        dict(kind="mirror", name="mirror_4x4x4", nx=4, ny=4, nz=4, steps=1),
        # static AMR: ghost fill in waves, coarse/fine corrections (470 active blocks)
        dict(kind="blast", name="blast_470", root=4, r0=0.4, r1=0.2, steps=16),
        # static AMR with gravity (594 active blocks on four levels)
        dict(kind="collapse", name="collapse_594", root=5, r0=0.4, r1=0.2, r2=0.1, steps=16),
        # a gradient through five steps: the backward direction
        dict(kind="adjoint", name="adjoint_4x4x4", nx=4, ny=4, nz=4, steps=5),
    ]


def draw(rng: random.Random):
    kind = rng.choice(["uniform"] * 6 + ["mirror", "blast", "collapse", "adjoint"])
    if kind == "blast":
        return dict(kind=kind, root=rng.choice([2, 3, 4]), r0=rng.uniform(0.2, 0.4), r1=rng.uniform(0.05, 0.18),
                    steps=rng.randint(3, 16))
    if kind == "collapse":
        return dict(kind=kind, root=rng.choice([3, 4, 5]), r0=rng.uniform(0.25, 0.4), r1=rng.uniform(0.12, 0.2),
                    r2=rng.uniform(0.05, 0.1), steps=rng.randint(3, 16))
    most = 512 if kind == "uniform" else 64
    n = int(round(math.exp(rng.uniform(math.log(8), math.log(most)))))
    nx = rng.randint(1, max(1, min(n, 16)))
    ny = rng.randint(1, max(1, min(n // nx, 16)))
    nz = max(1, min(n // (nx * ny), most // (nx * ny), 64))
    dims = [nx, ny, nz]
    rng.shuffle(dims)
    while dims[0] * dims[1] * dims[2] < 8:
        dims[dims.index(min(dims))] += 1
    c = dict(kind=kind, nx=dims[0], ny=dims[1], nz=dims[2])
    if kind == "mirror":
        return dict(c, steps=rng.randint(1, 3))
    if kind == "adjoint":
        return dict(c, steps=rng.randint(2, 5))
    c.update(mhd=rng.random() < 0.7, recon=rng.choice(["mc", "mc", "weno3"]),
             integrator=rng.choice(["rk2", "rk2", "rk2", "ess"]), form="batched")
    if dims[0] * dims[1] * dims[2] <= 40 and rng.random() < 0.4:
        c["form"] = "plain"
    c["steps"] = rng.randint(1, 2) if c["form"] == "plain" else rng.randint(1, 4) if c["integrator"] == "ess" \
        else rng.randint(2, 12 if c["recon"] == "mc" else 8)
    return c


# ---- inputs ---------------------------------------------------------------------

def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _modes(rng, n, kmax, amp):
    out = []
    for _ in range(n):
        k = [0, 0, 0]
        while not any(k):
            k = [rng.randint(-kmax, kmax) for _ in range(3)]
        d = [rng.gauss(0, 1) for _ in range(3)]
        dn = math.sqrt(sum(x * x for x in d))
        out.append((k, 2.0 * math.pi * rng.random(), [x / dn for x in d], amp / n))
    return out


def _sum(modes, x, y, z, comp=None):
    """Sum of the modes at x, y, z (any shapes that broadcast), or its
    component `comp` along the modes' directions."""
    s = None
    for k, ph, d, a in modes:
        c = torch.cos(2.0 * math.pi * (k[0] * x + k[1] * y + k[2] * z) + ph) * (a if comp is None else a * d[comp])
        s = c if s is None else s + c
    return s


def _dims(case):
    return case["nx"], case["ny"], case["nz"]


def _coord(case):
    """Cubic blocks, the longest side 1."""
    top = max(_dims(case))
    return [v for n in _dims(case) for v in (0.0, n / top)]


def _mhd(case):
    return case.get("mhd", True)


def _ess(case):
    return case.get("integrator", "rk2") == "ess"


def _global_state(case, seed):
    """Primitives [nv, X+4, Y+4, Z+4] (two ghost layers) and the face field
    (three arrays, one more along their own axis) of a uniform mesh."""
    rng = random.Random(seed * 7919 + 17)
    dev, mhd = _dev(), _mhd(case)
    gamma = 5.0 / 3.0
    n = _dims(case)
    h = 1.0 / (BS * max(n))
    amp = 0.1 if case["kind"] != "adjoint" else 0.01
    r, p = _modes(rng, 8, 4, amp), _modes(rng, 8, 4, amp)
    v, a = _modes(rng, 8, 4, amp), _modes(rng, 8, 4, 0.5 * amp)

    def axis(d, vertex):
        m = torch.arange(n[d] * BS + 2 * NG + (1 if vertex else 0), dtype=F8, device=dev) - NG
        s = (m + (0.0 if vertex else 0.5)) * h
        return s.reshape([-1 if q == d else 1 for q in range(3)])

    c = [axis(d, False) for d in range(3)]
    rho = 1.0 + _sum(r, *c)
    W = [rho] + [_sum(v, *c, comp=d) for d in range(3)]
    W += [(1.0 + _sum(p, *c)) / ((gamma - 1.0) * rho), 0.3 + 0.1 * _sum(r, *c)]
    B = None
    if mhd:
        A = [_sum(a, *[axis(q, q != d) for q in range(3)], comp=d) for d in range(3)]
        D = lambda x, d: torch.diff(x, dim=d) / h  # noqa: E731
        B = [D(A[2], 1) - D(A[1], 2), D(A[0], 2) - D(A[2], 0), D(A[1], 0) - D(A[0], 1)]
        W += _cell_b(B)
    return torch.stack(W), B


def _cell_b(B):
    m = [B[d].shape[d] - 1 for d in range(3)]
    return [0.5 * (B[d].narrow(d, 0, m[d]) + B[d].narrow(d, 1, m[d])) for d in range(3)]


def _blocks_of(a, extra=(0, 0, 0)):
    """Windows of the 16^3 blocks (with ghosts) of a global array, [blocks, ...]."""
    for d in range(3):
        a = a.unfold(d, P + extra[d], BS)
    return a.reshape(-1, *a.shape[3:])


def _face_extra(d):
    return tuple(1 if q == d else 0 for q in range(3))


def _pinned(shape):
    return torch.zeros(shape, dtype=F8, pin_memory=torch.cuda.is_available()).numpy()


@functools.lru_cache(maxsize=4)
def _amr_blocks(kind, root, *radii):
    hw = 0.7 if kind == "blast" else 1.0
    center = (0.1, 0.05, 0.0) if kind == "blast" else (0.0, 0.0, 0.0)
    coord = (-hw, hw, -hw, hw, -hw, hw)
    blocks = mesh.static_amr_mesh((root,) * 3, coord, len(radii), mesh.ball_refiner(center, radii))
    return blocks, mesh.to_desc(blocks), coord


def _amr_state(kind, blocks, coord, seed):
    """W [nb, 9, 20, 20, 20], Bf (three constants) and gravity of the AMR
    problems on every block entry."""
    rng = random.Random(seed * 104729 + 3)
    dev = _dev()
    lo = torch.tensor([b.xmin for b in blocks], dtype=F8, device=dev)
    dx = torch.tensor([b.dx for b in blocks], dtype=F8, device=dev)
    m = torch.arange(P, dtype=F8, device=dev) - NG + 0.5
    x, y, z = (lo[:, d].reshape(-1, 1, 1, 1) + m.reshape([1] + [-1 if q == d else 1 for q in range(3)]) *
               dx[:, d].reshape(-1, 1, 1, 1) for d in range(3))
    one = torch.ones(len(blocks), P, P, P, dtype=F8, device=dev)
    u = [rng.gauss(0, 1) for _ in range(3)]
    un = math.sqrt(sum(q * q for q in u))
    ripple = _sum(_modes(rng, 6, 3, 0.02), x, y, z)
    grav = None
    if kind == "blast":
        gamma = 5.0 / 3.0
        c = [0.1 + rng.uniform(-0.02, 0.02), 0.05 + rng.uniform(-0.02, 0.02), rng.uniform(-0.02, 0.02)]
        r = torch.sqrt((x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2)
        rho = one + ripple
        p = torch.where(r < 0.1, 10.0 * one, 0.1 * one)
        b0 = 1.0 / math.sqrt(4.0 * math.pi)
        vel = [0.0 * one] * 3
        eint = p / ((gamma - 1.0) * rho)
    else:
        gamma = 4.0 / 3.0
        rho_c, K, beta, r0 = 1.0e10, 4.6e5, 1.0e4, 0.1
        r = torch.sqrt(x * x + y * y + z * z)
        s = 1.0 + (r / r0) ** 2
        rho = rho_c / (s * torch.sqrt(s)) * (1.0 + ripple)
        p = K * rho ** gamma
        vr = -0.1 * torch.sqrt(gamma * p / rho) * r / (r + r0)
        inv = torch.where(r > 0, 1.0 / r, 0.0 * r)
        vel = [vr * q * inv for q in (x, y, z)]
        eint = p / ((gamma - 1.0) * rho)
        b0 = math.sqrt(2.0 * K * rho_c ** gamma / beta)
        q = r / r0
        menc = 4.0 * math.pi * rho_c * r0 ** 3 * (torch.asinh(q) - q / torch.sqrt(1.0 + q * q))
        g = torch.where(r > 0, -menc * inv ** 3, 0.0 * r)
        grav = torch.stack([(g * t + 0.0 * one) for t in (x, y, z)], 1)
    bf = [b0 * q / un for q in u]
    W = torch.stack([rho, *[q + 0.0 * one for q in vel], eint + 0.0 * one, 0.1 * one] + [b * one for b in bf], 1)
    return W, bf, grav, gamma


class State:
    """The context, its page-locked host arrays, the clock, and the views of
    the arrays' active region that a pass hands back."""

    def __init__(self, case):
        self.case = case
        self.clock = (0.0, 0.0, 0)

    def views(self, nb, nv, ns):
        a = slice(NG, NG + BS)
        f = slice(NG, NG + BS + 1)
        out = {"W": self.W.reshape(nb, nv, ns, P, P, P)[:, :, 0, a, a, a]}
        if self.Bf is not None:
            B = self.Bf.reshape(nb, 3, ns, -1)[:, :, 0]
            for d in range(3):
                shape = [P + (q == d) for q in range(3)]
                at = tuple(f if q == d else a for q in range(3))
                out["B%d" % (d + 1)] = B[:, d].reshape(nb, *shape)[(slice(None),) + at]
        self.out = out


def prepare(case, seed):
    st = State(case)
    kind = case["kind"]
    recon = fx.RECON_WENO3 if case.get("recon") == "weno3" else fx.RECON_MC
    integ = fx.INT_ESSPRK10_4 if _ess(case) else fx.INT_RK2
    grav = None
    if kind in ("blast", "collapse"):
        radii = [case[r] for r in ("r0", "r1", "r2") if r in case]
        blocks, desc, coord = _amr_blocks(kind, case["root"], *radii)
        nb, nv, mhd = len(blocks), 9, True
        W, bf, grav, gamma = _amr_state(kind, blocks, coord, seed)
        B = [torch.full((nb, P ** 2 * (P + 1)), b, dtype=F8) for b in bf]
    else:
        coord, mhd, gamma = _coord(case), _mhd(case), 5.0 / 3.0
        desc = mesh.to_desc(mesh.uniform_mesh(_dims(case), coord))
        nb, nv = len(desc), 9 if mhd else 6
        G, Bg = _global_state(case, seed)
        W = torch.stack([_blocks_of(G[v]) for v in range(nv)], 1)
        B = [_blocks_of(Bg[d], _face_extra(d)).reshape(nb, -1) for d in range(3)] if mhd else None
    ctx = fx.Context(mhd, gamma, coord, gravity=grav is not None, recon=recon, integrator=integ)
    ctx.set_mesh(desc)
    ns = ctx.ns
    st.W = _pinned((nb, nv, ns, P ** 3))
    torch.from_numpy(st.W)[:, :, :2] = W.reshape(nb, nv, 1, -1).cpu()
    st.Bf = None
    if mhd:
        st.Bf = _pinned((nb, 3, ns, P ** 2 * (P + 1)))
        for d in range(3):
            torch.from_numpy(st.Bf)[:, d, :2] = B[d].reshape(nb, 1, -1).cpu()
    ctx.upload_all(st.W, st.Bf)
    if grav is not None:
        g = grav.reshape(nb, 3, -1).cpu().numpy()
        for b in range(nb):
            ctx.upload_block(b, st.W[b], None, [g[b, d] for d in range(3)])
    ctx.boundary_fill(1, 0)
    ctx.sync()
    st.ctx = ctx
    if kind == "adjoint":
        # the objective's derivative at the final state: seeded weights of the active cells
        gen = torch.Generator().manual_seed(seed)
        bar = torch.zeros(nb, nv, ns, P, P, P, dtype=F8)
        a = slice(NG, NG + BS)
        bar[:, :, 0, a, a, a] = torch.randn(nb, nv, BS, BS, BS, dtype=F8, generator=gen)
        st.bar = bar.reshape(-1).numpy()
        st.dt = ctx.calc_dt(CFL)
    else:
        if case.get("form") != "plain":
            ctx.autotune()
        st.views(nb, nv, ns)
    return st


def run(state):
    case, ctx = state.case, state.ctx
    if case["kind"] == "adjoint":
        ctx.adjoint_forward(case["steps"], state.dt)
        W, B = ctx.adjoint_backward(state.bar)
        return {"W": W, "B": B}
    form = fx.FORM_PLAIN if case.get("form") == "plain" else fx.FORM_BATCHED
    if case["kind"] == "mirror":
        for _ in range(case["steps"]):
            ctx.upload_state_active(state.W, state.Bf)
            state.clock = ctx.run(form, 1, CFL, DT_FACTOR, T_END, state.clock)
            ctx.download_state_active(state.W, state.Bf)
    else:
        state.clock = ctx.run(form, case["steps"], CFL, DT_FACTOR, T_END, state.clock)
        ctx.download_state_active(state.W, state.Bf)
    return dict(state.out, t=state.clock[0], dt=state.clock[1], step=state.clock[2])


def work(case):
    """Bytes: per zone and step the variables read and written once per stage
    (72 B of 9 doubles, 48 B of 6: five passes per RK2 step), and what the
    host gets.  Flops: reconstruction and Riemann solve of three faces per
    zone and stage, edge EMFs and the cell update; a division or root counts
    as one."""
    if case["kind"] in ("blast", "collapse"):
        radii = [case[r] for r in ("r0", "r1", "r2") if r in case]
        nb = sum(b.active == 1 for b in _amr_blocks(case["kind"], case["root"], *radii)[0])
    else:
        nb = case["nx"] * case["ny"] * case["nz"]
    mhd = _mhd(case)
    z = nb * BS ** 3
    q = 72 if mhd else 48
    face = (450 if mhd else 220) + (500 if case.get("recon") == "weno3" else 0)
    stage = 3 * face + (250 if mhd else 80)
    stages, passes = (10, 10 * 2 + 2 * 2 + 3 * 3) if _ess(case) else (2, 5)
    s = case["steps"]
    if case["kind"] == "adjoint":
        # forward, every stage stored, and a reverse of about twice the work; the adjoint in and out
        return dict(bytes=s * z * q * (passes + 2 * stages + 2 * passes) + 2 * z * q, flops=3.0 * s * stages * stage * z)
    bytes_ = s * z * q * passes + z * q
    if case["kind"] == "mirror":
        bytes_ += (2 * s - 1) * z * q
    return dict(bytes=bytes_, flops=float(s * stages * stage * z))


def tolerance(case):
    # the framework's contract is the reference's own doubles, bit for bit;
    # the reverse sweep sums a cell's stencil adjoints in no fixed order
    return {"rel": 1e-13, "max": 1e-11} if case["kind"] == "adjoint" else "exact"


# ---- the same steps in plain torch ------------------------------------------------

def exact(case, seed):
    """One pass on a uniform mesh, restated on global arrays: None for the
    AMR problems and the reverse sweep."""
    if case["kind"] not in ("uniform", "mirror"):
        return None
    W, B = _global_state(case, seed)
    sim = _Plain(case, W, B)
    sim.fill()
    t, dt = 0.0, 0.0
    for _ in range(case["steps"]):
        new = sim.calc_dt()
        dt = min(new, DT_FACTOR * dt) if dt > 0 else new
        sim.step(dt)
        t += dt
    out = {"W": torch.stack([_act(_blocks_of(sim.W[v])) for v in range(len(sim.W))], 1)}
    for d in range(3 if sim.B else 0):
        out["B%d" % (d + 1)] = _act(_blocks_of(sim.B[d], _face_extra(d)))
    return dict(out, t=t, dt=dt, step=case["steps"])


def _act(b):
    return b[:, NG:-NG, NG:-NG, NG:-NG]


class _Plain:
    """RK2 / eSSPRK10_4 ideal MHD or hydro with outflow boundaries.  Arrays
    have two ghost layers; faces one more along their axis."""

    def __init__(self, case, W, B):
        self.n = [m * BS for m in _dims(case)]
        self.h = [(c1 - c0) / m for c0, c1, m in zip(_coord(case)[::2], _coord(case)[1::2], self.n)]
        self.g = 5.0 / 3.0
        self.mhd, self.ess, self.weno = _mhd(case), _ess(case), case.get("recon") == "weno3"
        self.W, self.B = list(W), B

    # boundaries: cells mirrored, faces continued
    def fill(self):
        dev = self.W[0].device
        for d in range(3):
            n = self.n[d]
            at = torch.arange(-NG, n + NG, device=dev)
            cell = torch.where(at < 0, -at - 1, torch.where(at >= n, 2 * n - 1 - at, at)) + NG
            self.W = [w.index_select(d, cell) for w in self.W]
            if self.mhd:
                near = at.clamp(0, n - 1) + NG
                face = torch.arange(-NG, n + NG + 1, device=dev).clamp(0, n) + NG
                self.B = [b.index_select(d, face if q == d else near) for q, b in enumerate(self.B)]
        if self.mhd:
            self.W[6:] = _cell_b(self.B)

    def _core(self, a):
        return a[NG:-NG, NG:-NG, NG:-NG]

    def calc_dt(self):
        w = [self._core(a) for a in self.W]
        cs = torch.sqrt(self.g * ((self.g - 1.0) * w[0] * w[4]) / w[0])
        s = (w[1].abs() + cs) / self.h[0] + (w[2].abs() + cs) / self.h[1] + (w[3].abs() + cs) / self.h[2]
        return float((CFL / s).min()) * (6.0 if self.ess else 1.0)

    def cons(self, w):
        ke = 0.5 * w[0] * (w[1] * w[1] + w[2] * w[2] + w[3] * w[3])
        e = w[0] * w[4] + ke
        if self.mhd:
            e = e + 0.5 * (w[6] * w[6] + w[7] * w[7] + w[8] * w[8])
        return [w[0], w[0] * w[1], w[0] * w[2], w[0] * w[3], e, w[0] * w[5]] + list(w[6:])

    def prim(self, u):
        v = [u[1] / u[0], u[2] / u[0], u[3] / u[0]]
        e = u[4] / u[0] - 0.5 * (v[0] * v[0] + v[1] * v[1] + v[2] * v[2])
        if self.mhd:
            e = e - 0.5 * (u[6] * u[6] + u[7] * u[7] + u[8] * u[8]) / u[0]
        return [u[0], *v, e, u[5] / u[0]] + list(u[6:])

    def step(self, dt):
        if not self.ess:
            W0, B0 = self.W, self.B
            self.euler(dt, None)
            self.euler(dt, (W0, B0, 0.5))
            return
        save = (self.W, self.B)
        for _ in range(5):
            self.euler(dt / 6.0, None)
        fifth = (self.W, self.B)
        self.blend(*save, 3.0 / 5.0)
        for _ in range(5):
            self.euler(dt / 6.0, None)
        self.blend(*fifth, 3.0 / 8.0)
        self.blend(*save, 1.0 / 25.0)

    def blend(self, W, B, w):
        if self.mhd:
            self.B = [w * b + (1.0 - w) * c for b, c in zip(B, self.B)]
        u = [w * a + (1.0 - w) * b for a, b in zip(self.cons(W), self.cons(self.W))]
        self.finish(u)

    def finish(self, u):
        if self.mhd:
            u[6:] = _cell_b(self.B)
        self.W = self.prim(u)
        self.fill()

    def euler(self, dt, avg):
        """One forward-Euler substep of the state; avg = (W0, B0, w): the
        average with that state (RK2's second stage)."""
        flux, emf = [], [None] * 3
        F = [self.faces(d) for d in range(3)]
        div = None
        for d in range(3):
            a = self.h[(d + 1) % 3] * self.h[(d + 2) % 3]
            t = [a * torch.diff(f, dim=d) for f in F[d][0]]
            div = t if div is None else [x + y for x, y in zip(div, t)]
        vol = self.h[0] * self.h[1] * self.h[2]
        if self.mhd:
            E = [self.edge(d, F) for d in range(3)]
            new = []
            for d in range(3):
                p, q = (d + 1) % 3, (d + 2) % 3
                b = self._faces_core(self.B[d], d)
                b = b - dt * torch.diff(E[q], dim=p) / self.h[p] + dt * torch.diff(E[p], dim=q) / self.h[q]
                if avg:
                    b = 0.5 * self._faces_core(avg[1][d], d) + 0.5 * b
                full = self.B[d].clone()
                self._faces_core(full, d).copy_(b)
                new.append(full)
            self.B = new
        u = self.cons(self.W)
        u0 = self.cons(avg[0]) if avg else None
        for v in range(6):
            x = self._core(u[v]) + dt * (-div[v] / vol)
            if avg:
                x = 0.5 * self._core(u0[v]) + 0.5 * x
            full = u[v].clone()
            self._core(full).copy_(x)
            u[v] = full
        self.finish(u)

    def _faces_core(self, b, d):
        return b[tuple(slice(NG, NG + self.n[q] + (q == d)) for q in range(3))]

    # reconstruction: states on both sides of the faces 0 .. n along d, one
    # ghost layer kept across
    def sides(self, a, d):
        n = self.n[d]
        for q in range(3):
            if q != d:
                a = a.narrow(q, 1, a.shape[q] - 2)
        q0, q1, q2, q3 = (a.narrow(d, m, n + 1) for m in range(4))
        if self.weno:
            return _weno3(q0, q1, q2, 0.5), _weno3(q1, q2, q3, -0.5)
        return q1 + 0.5 * _mc(q0, q1, q2), q2 - 0.5 * _mc(q1, q2, q3)

    def faces(self, d):
        """([six fluxes on the active faces], normal velocity and the two
        EMF products on the faces with their ring)."""
        m = [0] + [1 + (d + q) % 3 for q in range(3)] + [4, 5] + ([6 + (d + q) % 3 for q in range(3)] if self.mhd else [])
        pairs = {v: self.sides(self.W[v], d) for v in m if v != 6 + d}
        pairs["p"] = self.sides((self.g - 1.0) * self.W[0] * self.W[4], d)
        if self.mhd:
            bn = self.B[d]
            for q in range(3):
                bn = bn.narrow(q, NG, self.n[q] + 1) if q == d else bn.narrow(q, 1, bn.shape[q] - 2)
            pairs[6 + d] = (bn, bn)
        side = [dict(rho=pairs[0][s], u=pairs[m[1]][s], v=pairs[m[2]][s], w=pairs[m[3]][s], e=pairs[4][s],
                     ye=pairs[5][s], p=pairs["p"][s]) for s in range(2)]
        gl = gr = self.g
        if self.weno:
            one = torch.full((1,), self.g, dtype=F8, device=self.W[0].device)
            gl, gr = _weno3(one, one, one, 0.5), _weno3(one, one, one, -0.5)
        side[0]["g"], side[1]["g"] = gl, gr
        if self.mhd:
            for s in range(2):
                side[s].update(b=pairs[m[7]][s], c=pairs[m[8]][s])
            f, vn, e1, e2 = _hlld(side[0], side[1], pairs[6 + d][0])
        else:
            f, vn, e1, e2 = (*_hllc(side[0], side[1], *self.deltas(d)), None, None)
        out = [None] * 6
        for v, x in zip(m[:6], f):
            out[v] = x[tuple(slice(None) if q == d else slice(1, -1) for q in range(3))]
        return out, vn, e1, e2

    def deltas(self, d):
        """Velocity differences of the shock-shear limiter."""
        n = self.n

        def cut(a, off):
            for q in range(3):
                a = a.narrow(q, NG - 1 + off[q] if q == d else 1 + off[q], n[q] + 1 if q == d else n[q] + 2)
            return a

        def o(q, s):
            return [s if r == q else 0 for r in range(3)]

        un = self.W[1 + d]
        du = cut(un, o(d, 1)) - cut(un, o(d, 0))
        out = [du]
        for t in ((d + 1) % 3, (d + 2) % 3):
            x = self.W[1 + t]
            x = torch.nn.functional.pad(x, [v for q in (2, 1, 0) for v in ((1, 1) if q == t else (0, 0))])
            off = lambda dd, tt: [(dd if r == d else 0) + ((1 + tt) if r == t else 0) for r in range(3)]  # noqa: E731
            m = None
            for dd in (0, 1):
                c, lo, hi = cut(x, off(dd, 0)), cut(x, off(dd, -1)), cut(x, off(dd, 1))
                k = torch.minimum(c - lo, hi - c)
                m = k if m is None else torch.minimum(m, k)
            out.append(m)
        return out

    def edge(self, d, F):
        """Upwind EMF on the edges along d: active range 0 .. n across, n along."""
        up, rt = (d + 1) % 3, (d + 2) % 3
        w = self.W
        cell = w[6 + up] * w[1 + rt] - w[6 + rt] * w[1 + up]

        def at(a, ring, mu, mr):
            # a's value at edge - mu * up - mr * right; `ring`: ghost layers before index 0 per axis
            for q in range(3):
                m = mu if q == up else mr if q == rt else 0
                a = a.narrow(q, ring[q] - m, self.n[q] + (q != d))
            return a

        two = [NG] * 3
        ring = lambda nrm: [0 if q == nrm else 1 for q in range(3)]  # noqa: E731
        c = [at(cell, two, *s) for s in ((0, 0), (1, 0), (1, 1), (0, 1))]
        f = [at(F[rt][2], ring(rt), 0, 0), at(F[up][3], ring(up), 0, 0), at(F[rt][2], ring(rt), 1, 0),
             at(F[up][3], ring(up), 0, 1)]
        vn = [at(F[rt][1], ring(rt), 0, 0), at(F[up][1], ring(up), 0, 0), at(F[rt][1], ring(rt), 1, 0),
              at(F[up][1], ring(up), 0, 1)]
        e = 0.25 * (f[0] + f[1] + f[2] + f[3])
        for v, (fa, ca), (fb, cb) in ((vn[0], (3, 3), (1, 0)), (vn[1], (2, 1), (0, 0)), (vn[2], (3, 2), (1, 1)),
                                      (vn[3], (2, 2), (0, 3))):
            a, b = f[fa] - c[ca], f[fb] - c[cb]
            e = e + torch.where(v > 0, 0.25 * a, torch.where(v < 0, 0.25 * b, 0.125 * (f[fa] - c[ca] + f[fb] - c[cb])))
        return e


def _mc(a, b, c):
    l, r = b - a, c - b
    m = l + 0.5 * (r - l)
    s = torch.where(l > 0, torch.minimum(torch.minimum(2.0 * l, m), 2.0 * r),
                    torch.maximum(torch.maximum(2.0 * l, m), 2.0 * r))
    return torch.where(l * r > 0, s, 0.0 * s)


def _weno3(a, b, c, t):
    l, r = b - a, c - b
    p0, p1 = b + t * l, b + t * r
    b0, b1 = l * l, r * r
    tau = (b0 - b1).abs()
    g0, g1 = (1.0 / 3.0, 2.0 / 3.0) if t > 0 else (2.0 / 3.0, 1.0 / 3.0)
    a0 = g0 * (1.0 + tau / (1.0e-40 + b0))
    a1 = g1 * (1.0 + tau / (1.0e-40 + b1))
    return (a0 * p0 + a1 * p1) / (a0 + a1)


def _hllc(L, R, du, dv, dw):
    zero = torch.zeros_like(du)
    for s in (L, R):
        s["E"] = s["rho"] * s["e"] + 0.5 * s["rho"] * (s["u"] * s["u"] + s["v"] * s["v"] + s["w"] * s["w"])
        s["cs"] = torch.sqrt(s["g"] * s["p"] / s["rho"])
    SL = torch.minimum(L["u"] - L["cs"], R["u"] - R["cs"])
    SR = torch.maximum(L["u"] + L["cs"], R["u"] + R["cs"])
    cf = torch.maximum(L["cs"], R["cs"])
    th = (cf - torch.minimum(du, zero)) / (cf - torch.minimum(torch.minimum(dv, dw), zero))
    th = th * th
    th = torch.minimum(torch.ones_like(th), th * th)
    mL, mR = L["rho"] * (SL - L["u"]), R["rho"] * (SR - R["u"])
    SM = (th * (R["p"] - L["p"]) + L["rho"] * L["u"] * (SL - L["u"]) - R["rho"] * R["u"] * (SR - R["u"])) / (mL - mR)

    def side(s, S, m):
        U = [s["rho"], s["rho"] * s["u"], s["rho"] * s["v"], s["rho"] * s["w"], s["E"], s["rho"] * s["ye"]]
        F = [U[1], U[1] * s["u"] + s["p"], U[1] * s["v"], U[1] * s["w"], (s["E"] + s["p"]) * s["u"], U[5] * s["u"]]
        r = m / (S - SM)
        e = s["E"] / s["rho"] + (SM - s["u"]) * (SM + s["p"] / m)
        V = [r, r * SM, r * s["v"], r * s["w"], r * e, r * s["ye"]]
        return F, [f + S * (v - u) for f, v, u in zip(F, V, U)]

    FL, GL = side(L, SL, mL)
    FR, GR = side(R, SR, mR)

    def pick(a, b, c, d):
        return torch.where(SL >= 0, a, torch.where(SR <= 0, b, torch.where(SM >= 0, c, d)))

    return [pick(*q) for q in zip(FL, FR, GL, GR)], pick(L["u"], R["u"], SM, SM)


def _hlld(L, R, bn):
    for s in (L, R):
        s["bt"] = 0.5 * (bn * bn + s["b"] * s["b"] + s["c"] * s["c"])
        s["E"] = s["rho"] * s["e"] + 0.5 * s["rho"] * (s["u"] * s["u"] + s["v"] * s["v"] + s["w"] * s["w"]) + s["bt"]
        s["P"] = s["p"] + s["bt"]
        a2, x2, b2 = s["g"] * s["p"] / s["rho"], bn * bn / s["rho"], (bn * bn + s["b"] * s["b"] + s["c"] * s["c"]) / s["rho"]
        disc = ((a2 + b2) * (a2 + b2) - 4.0 * a2 * x2).clamp(min=0.0)
        s["cf"] = torch.sqrt(0.5 * (a2 + b2 + torch.sqrt(disc)))
    SL = torch.minimum(L["u"] - L["cf"], R["u"] - R["cf"])
    SR = torch.maximum(L["u"] + L["cf"], R["u"] + R["cf"])
    mL, mR = L["rho"] * (SL - L["u"]), R["rho"] * (SR - R["u"])
    SM = (R["rho"] * R["u"] * (SR - R["u"]) - L["rho"] * L["u"] * (SL - L["u"]) + (L["P"] - R["P"])) / (mR - mL)
    pt = 0.5 * ((L["P"] + mL * (SM - L["u"])) + (R["P"] + mR * (SM - R["u"])))

    def outer(s, S):
        al, sm = S - s["u"], S - SM
        r = s["rho"] * al / sm
        den = s["rho"] * al * sm - bn * bn
        flat = den.abs() < 1.0e-8 * pt
        k, m = (SM - s["u"]) / den, (s["rho"] * al * al - bn * bn) / den
        v = torch.where(flat, s["v"], s["v"] - bn * s["b"] * k)
        w = torch.where(flat, s["w"], s["w"] - bn * s["c"] * k)
        b, c = torch.where(flat, s["b"], s["b"] * m), torch.where(flat, s["c"], s["c"] * m)
        vb, vb1 = s["u"] * bn + s["v"] * s["b"] + s["w"] * s["c"], SM * bn + v * b + w * c
        E = (al * s["E"] - s["P"] * s["u"] + pt * SM + bn * (vb - vb1)) / sm
        return dict(rho=r, u=SM, v=v, w=w, b=b, c=c, E=E, ye=s["ye"])

    def cons(s):
        return [s["rho"], s["rho"] * s["u"], s["rho"] * s["v"], s["rho"] * s["w"], s["E"], s["rho"] * s["ye"]]

    def flux(s):
        m = s["rho"] * s["u"]
        vb = s["u"] * bn + s["v"] * s["b"] + s["w"] * s["c"]
        return [m, m * s["u"] + s["P"] - bn * bn, m * s["v"] - bn * s["b"], m * s["w"] - bn * s["c"],
                (s["E"] + s["P"]) * s["u"] - bn * vb, s["rho"] * s["ye"] * s["u"]]

    def out(s):
        return [s["u"], s["c"] * s["u"] - bn * s["w"], bn * s["v"] - s["b"] * s["u"]]

    Ls, Rs = outer(L, SL), outer(R, SR)
    ql, qr = torch.sqrt(Ls["rho"]), torch.sqrt(Rs["rho"])
    SLs, SRs = SM - bn.abs() / ql, SM + bn.abs() / qr
    sg = torch.where(bn < 0, -torch.ones_like(bn), torch.ones_like(bn))
    inv = 1.0 / (ql + qr)
    mid = dict(u=SM, v=(ql * Ls["v"] + qr * Rs["v"] + (Rs["b"] - Ls["b"]) * sg) * inv,
               w=(ql * Ls["w"] + qr * Rs["w"] + (Rs["c"] - Ls["c"]) * sg) * inv,
               b=(ql * Rs["b"] + qr * Ls["b"] + ql * qr * (Rs["v"] - Ls["v"]) * sg) * inv,
               c=(ql * Rs["c"] + qr * Ls["c"] + ql * qr * (Rs["w"] - Ls["w"]) * sg) * inv)
    vb = SM * bn + mid["v"] * mid["b"] + mid["w"] * mid["c"]

    def dbl(s, q, sign):
        vs = SM * bn + s["v"] * s["b"] + s["w"] * s["c"]
        return dict(s, E=s["E"] + sign * (q * sg * (vs - vb)), **mid)

    Ld, Rd = dbl(Ls, ql, -1.0), dbl(Rs, qr, 1.0)
    UL, UR, ULs, URs, FL, FR = cons(L), cons(R), cons(Ls), cons(Rs), flux(L), flux(R)
    left = SM >= 0
    small = 0.5 * bn * bn < 1.0e-8 * pt
    one_l, one_r = (SLs >= 0) | small, (SRs <= 0) | small

    def pick(a, b, ls, rs, ld, rd):
        star = torch.where(left, torch.where(one_l, ls, ld), torch.where(one_r, rs, rd))
        return torch.where(SL >= 0, a, torch.where(SR <= 0, b, star))

    F = []
    for v, (ld, rd) in enumerate(zip(cons(Ld), cons(Rd))):
        ls, rs = FL[v] + SL * (ULs[v] - UL[v]), FR[v] + SR * (URs[v] - UR[v])
        F.append(pick(FL[v], FR[v], ls, rs, ls + SLs * (ld - ULs[v]), rs + SRs * (rd - URs[v])))
    o = [pick(*q) for q in zip(out(L), out(R), out(Ls), out(Rs), out(Ld), out(Rd))]
    return [F, *o]
