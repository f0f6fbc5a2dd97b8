/*
 * Per-phase kernels of the RK2 Godunov MHD update, one thread per face, edge
 * or cell.  Every kernel takes a block list: the plain (drop-in) form passes
 * one block per launch, as the reference's per-block loops do; the batched
 * form passes every block of the mesh in one launch.
 *
 * Phase                       reference
 * face fluxes (k_flux)        prj_flux_update, src/prj_flux.c:2149-2521
 * edge EMFs (k_emf)           prj_timeint_mhd_update_emf, src/prj_timeint.c:292-413
 * CT face update (k_bf_update) prj_timeint_mhd_update_bf, src/prj_timeint.c:415-495
 * cell update (k_cell_update) src/prj_timeint.c:1255-1349 and 1562-1654,
 *                             src terms src/prj_src.c:32-139, 717-768
 * eos fill (k_eos_fill)       prj_eos_fill_block/_active_cells, src/prj_eos.c:1087-1162
 * dt (k_calc_dt)              prj_timeint_calc_dt, src/prj_timeint.c:2144-2256
 * ghost programs              prj_boundary_fill_ghosts_and_bf, src/prj_boundary.c:1150-1241
 * bf2bc                       prj_mhd_bf2bc_impl, src/prj_mhd.c:555-603: ghost cells in
 *                             the ghost programs, active cells in k_cell_field_active
 */
#include <cuda_runtime.h>

#include <type_traits>

#include "../../include/fornax_b200.h"
#include "fx_kernels.h"
#include "fx_physics.cuh"

namespace {

constexpr int kPlane = FX_NSTAGES * FX_NCELLS; /* stride between variables of W */

/* the face arrays take no more memory than the reference's tiles would */
static_assert(FX_CF_COUNT + FX_CX_COUNT + FX_VN_COUNT + FX_VT_COUNT <= (3 * 9 + 9) * FX_NCELLS, "MHD");
static_assert(FX_CF_COUNT + FX_VN_COUNT + FX_VT_COUNT <= (3 * 6 + 9) * FX_NCELLS, "hydro");

__device__ __forceinline__ int fx_axis_stride(int dir)
{
    return dir == 0 ? FX_PBS * FX_PBS : dir == 1 ? FX_PBS : 1;
}

/* local (sweep-rotated) variable -> global variable, prj_flux_build_var_map
 * (src/prj_flux.c:274-349): the sweep-normal velocity and field go to slot 1
 * and 6 of the local vector. */
__device__ __forceinline__ int fx_gmap(int dir, int lv)
{
    if (lv >= 1 && lv <= 3) {
        return 1 + (dir + lv - 1) % 3;
    }
    if (lv >= 6) {
        return 6 + (dir + lv - 6) % 3;
    }
    return lv;
}

__device__ __forceinline__ unsigned long long fx_double_key(double d)
{
    unsigned long long bits = (unsigned long long)__double_as_longlong(d);
    return (bits >> 63) ? ~bits : (bits | 0x8000000000000000ULL);
}

/* ------------------------------------------------------------------------ */
/* Face fluxes                                                               */
/* ------------------------------------------------------------------------ */
/* MC face values of a 4-cell stencil with the limiter's selections through
 * a branch policy: bits 4 q + 0 and 4 q + 2 of the face's word */
template <class BR>
__device__ __forceinline__ void fx_recon_pair_br(const double (&q)[4], double &wl, double &wr, BR &br, int q4)
{
    wl = q[1] + 0.5 * fx_mc_slope_br(q[0], q[1], q[2], br, q4);
    wr = q[2] - 0.5 * fx_mc_slope_br(q[1], q[2], q[3], br, q4 + 2);
}

/* a stencil value of the face kernel: through the read-only data path for
 * the 4-cell stencils (MC, WENO-Z3), a plain load for WENO-Z7's 8 cells */
template <int RECON>
__device__ __forceinline__ double fx_stencil_load(const double *p)
{
    if constexpr (RECON == FX_RECON_WENO7) {
        return *p;
    } else {
        return __ldg(p);
    }
}

/* A face whose cheap checks did not pass (FxSuspect), evaluated again with
 * the solver's checks themselves: reports the first that fails, if one does.
 * Out of line: no sound state comes here.  q0: first stencil cell of
 * variable 0; bnp: the face's normal field. */
template <int RECON>
__device__ __noinline__ void fx_face_recheck(FxErr *err, const double *q0, const double *bnp, int dir, int s,
    double g, double gL, double gR, int b, int cR)
{
    constexpr int NS = FxStencil<RECON>::NS;
    double WL[9], WR[9], pS[NS], pL, pR;
    for (int lv = 0; lv < 9; ++lv) {
        if (lv == FX_B1) {
            WL[lv] = *bnp;
            WR[lv] = *bnp;
            continue;
        }
        const double *q = q0 + (size_t)fx_gmap(dir, lv) * kPlane;
        double qs[NS];
        for (int n = 0; n < NS; ++n) qs[n] = q[n * s];
        fx_recon_pair<RECON>(qs, WL[lv], WR[lv]);
    }
    for (int n = 0; n < NS; ++n) {
        pS[n] = fx_pressure(g, q0[(size_t)FX_RHO * kPlane + n * s], q0[(size_t)FX_EINT * kPlane + n * s]);
    }
    fx_recon_pair<RECON>(pS, pL, pR);
    FxErrLocal le;
    FxBrFree br;
    FxFaceOut o;
    fx_riemann_hlld_folded_br(WL, WR, pL, pR, gL, gR, *bnp, o, &le, b, cR, br);
    if (le.code != 0) {
        fx_fail(err, le.code, le.block, le.index);
    }
}

/* The faces of one sweep direction: DIR, or blockIdx.y's if DIR is -1.  With a
 * compile-time direction the strides, rotated variables and output planes are
 * immediate offsets, but the kernel holds three copies of the body, run side by
 * side.  Hydro gains (216 blocks 106 -> 92 us); three MHD bodies overrun the
 * instruction cache (512 blocks 503 -> 583 us; with the directions one after
 * the other 525 us, the stencils then read from DRAM three times). */
template <bool MHD, bool FULL, bool RING, int TPB, int RECON, int BRM, int DIR, class Br>
__device__ __forceinline__ void fx_flux_dir(const FxDev &D, const int *__restrict__ blist, int wslot, int bfslot,
    double gL, double gR, Br &br)
{
    const int dir = DIR < 0 ? (int)blockIdx.y : DIR;
    /* grid (face chunk, direction, block): the three sweeps of a block are
     * scheduled back to back, so its stencil cells are re-read from L2 */
    const int b = blist[blockIdx.z];
    /* MHD carries one transverse ghost layer of faces for the CT EMFs
     * (src/prj_flux.c:2241-2251); hydro transverse faces are [0, 15]. */
    constexpr int T = MHD ? FX_BS + 2 : FX_BS;
    constexpr int TLO = MHD ? -1 : 0;
    constexpr int NF = (FX_BS + 1) * T * T;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= NF) {
        return;
    }
    /* this face's decision word (record / replay) */
    const size_t bri = D.br_off + ((size_t)b * 3 + dir) * NF + t;
    if constexpr (BRM == 2) {
        br.w = D.br_words[bri];
    }
    const int e2 = dir == 2 ? FX_BS + 1 : T;
    const int e1 = dir == 1 ? FX_BS + 1 : T;
    const int k = (dir == 2 ? 0 : TLO) + t % e2;
    t /= e2;
    const int j = (dir == 1 ? 0 : TLO) + t % e1;
    const int i = (dir == 0 ? 0 : TLO) + t / e1;
    const int s = fx_axis_stride(dir);
    const int cR = fx_lidx(i, j, k);
    const int cL = cR - s;
    const int nv = MHD ? 9 : 6;
    const double *Wb = D.W + (size_t)b * FX_W_COUNT(nv) + (size_t)wslot * FX_NCELLS;
    const double g = D.gamma;

    double WL[9];
    double WR[9];
    /* the MHD solver takes the internal energy and composition of one side
     * only and asks for them when it knows which: worth its late loads for
     * the WENO values (WENO-Z3, 216 blocks: 490 -> 470 us), not for two MC
     * slopes (512 blocks: 503 -> 551 us) */
    constexpr bool kLazy = MHD && BRM == 0 && RECON != FX_RECON_MC;
    /* density and internal energy at the stencil cells also give the
     * reconstructed pressure (eosvar p = (g-1) rho e of each cell).  The
     * MC and WENO-Z3 stencils come through the read-only data path
     * (fx_stencil_load): this launch does not write W (on the 128^3 state
     * 0.628 -> 0.623 ms at 64 x 8, 0.699 -> 0.665 ms at 256 x 3; the normal
     * field that way, and the EMF, CT, fill and cell kernels, measured no
     * faster; WENO-Z7's 8-cell stencils 4.60 ms with plain loads against
     * 4.75 ms). */
    constexpr int NS = FxStencil<RECON>::NS;
    const int c0 = cL - (NS / 2 - 1) * s;   /* first stencil cell */
    double rhoS[NS], eintS[NS];
    {
        const double *qr = Wb + (size_t)FX_RHO * kPlane + c0;
        const double *qe = Wb + (size_t)FX_EINT * kPlane + c0;
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            rhoS[n] = fx_stencil_load<RECON>(qr + n * s);
            eintS[n] = fx_stencil_load<RECON>(qe + n * s);
        }
    }
    if constexpr (BRM == 0) {
        fx_recon_pair<RECON>(rhoS, WL[FX_RHO], WR[FX_RHO]);
        if constexpr (!kLazy) {
            fx_recon_pair<RECON>(eintS, WL[FX_EINT], WR[FX_EINT]);
        }
    } else {
        fx_recon_pair_br(rhoS, WL[FX_RHO], WR[FX_RHO], br, 4 * FX_RHO);
        fx_recon_pair_br(eintS, WL[FX_EINT], WR[FX_EINT], br, 4 * FX_EINT);
    }
#pragma unroll
    for (int lv = 1; lv < nv; ++lv) {
        if (lv == FX_EINT || (MHD && lv == FX_B1) || (kLazy && lv == FX_YE)) {
            continue;
        }
        const double *q = Wb + (size_t)fx_gmap(dir, lv) * kPlane + c0;
        double qs[NS];
#pragma unroll
        for (int n = 0; n < NS; ++n) {
            qs[n] = fx_stencil_load<RECON>(q + n * s);
        }
        if constexpr (BRM == 0) {
            fx_recon_pair<RECON>(qs, WL[lv], WR[lv]);
        } else {
            fx_recon_pair_br(qs, WL[lv], WR[lv], br, 4 * lv);
        }
    }
    double pS[NS];
#pragma unroll
    for (int n = 0; n < NS; ++n) {
        pS[n] = fx_pressure(g, rhoS[n], eintS[n]);
    }
    double pL, pR;
    if constexpr (BRM == 0) {
        fx_recon_pair<RECON>(pS, pL, pR);
    } else {
        /* the pressure takes the normal field's (unreconstructed) bits */
        fx_recon_pair_br(pS, pL, pR, br, 4 * FX_B1);
    }
    /* the transverse velocities of the plain form */
    double *vt = D.vt + (size_t)b * FX_VT_COUNT + (size_t)dir * 2 * FX_NCELLS + cR;
    if (MHD) {
        const double *bnp = D.Bf + (size_t)b * FX_BF_COUNT + ((size_t)dir * FX_NSTAGES + bfslot) * FX_NFACES +
            fx_face_idx(dir, i, j, k);
        const double bn = *bnp;
        FxSuspect suspect;
        WL[FX_B1] = bn;
        WR[FX_B1] = bn;
        FxFaceOut o;
        if constexpr (BRM == 0) {
            FxBrFree bf;
            if constexpr (kLazy) {
                fx_riemann_hlld_folded_br(WL, WR, pL, pR, gL, gR, bn, o, &suspect, b, cR, bf,
                    [q0 = Wb + c0, s](bool left, double &eint, double &ye) {
                        eint = fx_recon_one<RECON>(q0 + (size_t)FX_EINT * kPlane, s, left);
                        ye = fx_recon_one<RECON>(q0 + (size_t)FX_YE * kPlane, s, left);
                    });
            } else {
                fx_riemann_hlld_folded_br(WL, WR, pL, pR, gL, gR, bn, o, &suspect, b, cR, bf);
            }
        } else {
            fx_riemann_hlld_folded_br(WL, WR, pL, pR, gL, gR, bn, o, D.err, b, cR, br);
            if constexpr (BRM == 1) {
                D.br_words[bri] = br.w;
            } else if (br.flips) {
                atomicAdd(D.br_flips, (unsigned long long)br.flips);
            }
        }
        const bool own = fx_is_face(dir, 0, i, j, k); /* the ghost layer serves the EMFs only */
        if (RING || own) {
            double *f = own ? D.cf + (size_t)b * FX_CF_COUNT + fx_cf_idx(dir, i, j, k)
                            : D.cx + (size_t)b * FX_CX_COUNT + fx_cx_idx(dir, i, j, k);
            const int plane = own ? fx_cf_plane(dir) : fx_cx_plane(dir);
#pragma unroll
            for (int lv = 0; lv < 6; ++lv) {
                f[fx_gmap(dir, lv) * plane] = o.F[lv];
            }
        }
        const size_t bvi = (size_t)b * FX_BV_COUNT + (size_t)dir * FX_NCELLS + cR;
        D.vn[bvi] = o.v[0];
        if constexpr (FULL) {
#pragma unroll
            for (int lv = 6; lv < 9; ++lv) {
                D.cx[(size_t)b * FX_CX_COUNT + fx_cx_field(dir, fx_gmap(dir, lv), i, j, k)] = o.F[lv];
            }
            vt[0] = o.v[1];
            vt[FX_NCELLS] = o.v[2];
        }
        D.bv1[bvi] = o.bv1;
        D.bv2[bvi] = o.bv2;
        if constexpr (BRM == 0) {
            if (suspect.any) {
                fx_face_recheck<RECON>(D.err, Wb + c0, bnp, dir, s, g, gL, gR, b, cR);
            }
        }
    } else {
        /* transverse velocity deltas of the theta limiter,
         * prj_flux_velocity_deltas (src/prj_flux.c:1967-2036) */
        const int da = (dir + 1) % 3;
        const int db = (dir + 2) % 3;
        const int sa = fx_axis_stride(da);
        const int sb = fx_axis_stride(db);
        const double *un = Wb + (size_t)(1 + dir) * kPlane;
        const double *ua = Wb + (size_t)(1 + da) * kPlane;
        const double *ub = Wb + (size_t)(1 + db) * kPlane;
        const double du = un[cR] - un[cL];
        const double dv = fx_min(fx_min(ua[cL] - ua[cL - sa], ua[cL + sa] - ua[cL]),
            fx_min(ua[cR] - ua[cR - sa], ua[cR + sa] - ua[cR]));
        const double dw = fx_min(fx_min(ub[cL] - ub[cL - sb], ub[cL + sb] - ub[cL]),
            fx_min(ub[cR] - ub[cR - sb], ub[cR + sb] - ub[cR]));
        double F[6];
        double v[3];
        fx_riemann_hllc(WL, WR, pL, pR, gL, gR, du, dv, dw, F, v);
        double *cf = D.cf + (size_t)b * FX_CF_COUNT + fx_cf_idx(dir, i, j, k);
        const int plane = fx_cf_plane(dir);
#pragma unroll
        for (int lv = 0; lv < 6; ++lv) {
            cf[fx_gmap(dir, lv) * plane] = F[lv];
        }
        D.vn[(size_t)b * FX_VN_COUNT + (size_t)dir * FX_NCELLS + cR] = v[0];
        if constexpr (FULL) {
            vt[0] = v[1];
            vt[FX_NCELLS] = v[2];
        }
    }
}

/* FULL: store every component the reference stores (the drop-in form);
 * otherwise only what later phases read (hydro flux components, the normal
 * face velocity, Bv1/Bv2).  TPB/MINB set the launch shape (threads per CTA,
 * resident CTAs per SM the register allocation must allow); the autotuner
 * picks among the compiled shapes.
 * BRM: 0 the solver as it stands; 1 record / 2 replay every face's
 * decisions in D.br_words (FxBrRecord / FxBrReplay; MHD, MC and the plain
 * form only), the branch-frozen map the adjoint checks use.
 * RING (MHD): the fluxes of the transverse ghost layer are stored too.
 * Downloads alone read them, and they cost a launch 500 -> 541 us at 512
 * blocks, so only the last launch of a call has them.  A kernel of its own:
 * with the store behind a run-time test the launches without it take 522 us,
 * with both bodies in one kernel a run of 105 blocks 0.8 % longer. */
template <bool MHD, bool FULL, bool RING, int TPB, int MINB, int RECON, int BRM = 0>
__global__ void __launch_bounds__(TPB, MINB) k_flux(FxDev D, const int *__restrict__ blist,
    int wslot, int bfslot)
{
    static_assert(BRM == 0 || (MHD && FULL && RECON == FX_RECON_MC), "decision record / replay: MHD, MC, plain");
    using Br = typename std::conditional<BRM == 1, FxBrRecord,
        typename std::conditional<BRM == 2, FxBrReplay, FxBrFree>::type>::type;
    Br br;
    if (D.ctl->skip) {
        return;
    }
    /* gamma is uniform for the ideal gas: its MC slope is exactly 0, so the
     * MC face values equal g bit for bit; the WENO weights of a constant
     * stencil are evaluated as the reference does (their sum need not be 1).
     * Those face values depend on g alone, so one thread of the CTA
     * evaluates them for all (before any thread leaves). */
    __shared__ double s_gface[2];
    if constexpr (RECON != FX_RECON_MC) {
        if (threadIdx.x == 0) {
            double gS[FxStencil<RECON>::NS];
#pragma unroll
            for (int n = 0; n < FxStencil<RECON>::NS; ++n) {
                gS[n] = D.gamma;
            }
            fx_recon_pair<RECON>(gS, s_gface[0], s_gface[1]);
        }
        __syncthreads();
    }
    double gL = D.gamma, gR = D.gamma;
    if constexpr (RECON != FX_RECON_MC) {
        gL = s_gface[0];
        gR = s_gface[1];
    }
    if constexpr (MHD) {
        fx_flux_dir<MHD, FULL, RING, TPB, RECON, BRM, -1>(D, blist, wslot, bfslot, gL, gR, br);
    } else {
        switch (blockIdx.y) {
        case 0: fx_flux_dir<MHD, FULL, RING, TPB, RECON, BRM, 0>(D, blist, wslot, bfslot, gL, gR, br); break;
        case 1: fx_flux_dir<MHD, FULL, RING, TPB, RECON, BRM, 1>(D, blist, wslot, bfslot, gL, gR, br); break;
        default: fx_flux_dir<MHD, FULL, RING, TPB, RECON, BRM, 2>(D, blist, wslot, bfslot, gL, gR, br); break;
        }
    }
}

/* ------------------------------------------------------------------------ */
/* Edge EMFs                                                                 */
/* ------------------------------------------------------------------------ */
/* The per-block launches of the plain form: one thread per edge, so a
 * single block still fills the device; the cell EMF components and eta of
 * an edge's four cells are evaluated per edge (same arithmetic). */
__device__ __forceinline__ double fx_cell_emf(const double *Wb, int dir, int c)
{
    const int a = (dir + 1) % 3;
    const int bb = (dir + 2) % 3;
    const double bA = Wb[(size_t)(FX_B1 + a) * kPlane + c];
    const double bB = Wb[(size_t)(FX_B1 + bb) * kPlane + c];
    const double vA = Wb[(size_t)(FX_V1 + a) * kPlane + c];
    const double vB = Wb[(size_t)(FX_V1 + bb) * kPlane + c];
    return bA * vB - bB * vA;
}

/* the plain form, and the batched form on a short list */
__global__ void __launch_bounds__(128) k_emf_edges(FxDev D, const int *__restrict__ blist, int wslot, int bfslot)
{
    if (D.ctl->skip) {
        return;
    }
    const int b = blist[blockIdx.y];
    constexpr int NE = FX_BS * (FX_BS + 1) * (FX_BS + 1);
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * NE) {
        return;
    }
    const int dir = t / NE;
    t -= dir * NE;
    const int te = t; /* edge index within the direction */
    const int x2 = dir == 2 ? FX_BS : FX_BS + 1;
    const int x1 = dir == 1 ? FX_BS : FX_BS + 1;
    int e[3];
    e[2] = t % x2;
    t /= x2;
    e[1] = t % x1;
    e[0] = t / x1;
    const int up = (dir + 1) % 3;
    const int right = (dir + 2) % 3;
    const int su = fx_axis_stride(up);
    const int sr = fx_axis_stride(right);
    const int c0 = fx_lidx(e[0], e[1], e[2]);   /* cell0 = e; face0 = face1 = e */
    const int c1 = c0 - su;                      /* cell1 = e - up */
    const int c2 = c0 - su - sr;                 /* cell2 = e - up - right */
    const int c3 = c0 - sr;                      /* cell3 = e - right */
    const double *Wb = D.W + (size_t)b * FX_W_COUNT(9) + (size_t)wslot * FX_NCELLS;
    const double *bv1r = D.bv1 + (size_t)b * FX_BV_COUNT + (size_t)right * FX_NCELLS;
    const double *bv2u = D.bv2 + (size_t)b * FX_BV_COUNT + (size_t)up * FX_NCELLS;
    const double *vnr = D.vn + (size_t)b * FX_VN_COUNT + (size_t)right * FX_NCELLS;
    const double *vnu = D.vn + (size_t)b * FX_VN_COUNT + (size_t)up * FX_NCELLS;
    double f[4], c[4], vn[4];
    /* face0 = e (right-normal), face1 = e (up-normal), face2 = e - up
     * (right-normal), face3 = e - right (up-normal) */
    f[0] = bv1r[c0];
    f[1] = bv2u[c0];
    f[2] = bv1r[c1];
    f[3] = bv2u[c3];
    c[0] = fx_cell_emf(Wb, dir, c0);
    c[1] = fx_cell_emf(Wb, dir, c1);
    c[2] = fx_cell_emf(Wb, dir, c2);
    c[3] = fx_cell_emf(Wb, dir, c3);
    vn[0] = vnr[c0];
    vn[1] = vnu[c0];
    vn[2] = vnr[c1];
    vn[3] = vnu[c3];
    const int eidx = fx_edge_idx(dir, e[0], e[1], e[2]);
    for (int n = 0; n < 4; ++n) {
        if (!isfinite(f[n]) || !isfinite(c[n]) || !isfinite(vn[n])) {
            fx_fail(D.err, FX_ERR_EMF_NONFINITE, b, eidx);
        }
    }
    /* edge resistivity: run-time eta plus the maximum artificial eta of the
     * four incident cells (src/prj_timeint.c:265-290) */
    double eta_cells = 0.0;
    {
        const int cells[4] = {c0, c1, c2, c3};
        for (int n = 0; n < 4; ++n) {
            const double ce = fx_cell_eta(Wb[(size_t)FX_RHO * kPlane + cells[n]],
                Wb[(size_t)FX_YE * kPlane + cells[n]]);
            if (!isfinite(ce) || ce < 0.0) {
                fx_fail(D.err, FX_ERR_ETA, b, eidx);
            }
            if (ce > eta_cells) {
                eta_cells = ce;
            }
        }
    }
    const double eta = D.mhd_eta + eta_cells;
    double emf;
    if (D.br_mode == 0) {
        emf = fx_emf_upwind(f, c, vn);
    } else {
        /* this edge's decision word (record / replay) */
        const size_t bri = D.br_eoff + ((size_t)b * 3 + dir) * NE + te;
        if (D.br_mode == 1) {
            FxBrRecord br;
            emf = fx_emf_upwind_br(f, c, vn, br);
            D.br_edges[bri] = br.w;
        } else {
            FxBrReplay br;
            br.w = D.br_edges[bri];
            emf = fx_emf_upwind_br(f, c, vn, br);
            if (br.flips) {
                atomicAdd(D.br_flips, (unsigned long long)br.flips);
            }
        }
    }
    if (eta != 0.0) {
        /* resistive term, src/prj_mhd.c:682-709 */
        const double *bf = D.Bf + (size_t)b * FX_BF_COUNT;
        const double *b1 = bf + (size_t)(0 * FX_NSTAGES + bfslot) * FX_NFACES;
        const double *b2 = bf + (size_t)(1 * FX_NSTAGES + bfslot) * FX_NFACES;
        const double *b3 = bf + (size_t)(2 * FX_NSTAGES + bfslot) * FX_NFACES;
        const FxBlockDev &B = D.blk[b];
        const int i = e[0], j = e[1], k = e[2];
        double curl_b;
        if (dir == 0) {
            curl_b = (b3[fx_face_idx(2, i, j, k)] - b3[fx_face_idx(2, i, j - 1, k)]) / B.dx[1] -
                (b2[fx_face_idx(1, i, j, k)] - b2[fx_face_idx(1, i, j, k - 1)]) / B.dx[2];
        } else if (dir == 1) {
            curl_b = (b1[fx_face_idx(0, i, j, k)] - b1[fx_face_idx(0, i, j, k - 1)]) / B.dx[2] -
                (b3[fx_face_idx(2, i, j, k)] - b3[fx_face_idx(2, i - 1, j, k)]) / B.dx[0];
        } else {
            curl_b = (b2[fx_face_idx(1, i, j, k)] - b2[fx_face_idx(1, i - 1, j, k)]) / B.dx[0] -
                (b1[fx_face_idx(0, i, j, k)] - b1[fx_face_idx(0, i, j - 1, k)]) / B.dx[1];
        }
        emf += eta * curl_b;
    }
    if (!isfinite(emf)) {
        fx_fail(D.err, FX_ERR_EMF_NONFINITE, b, eidx);
    }
    D.emf[(size_t)b * FX_EMF_COUNT + (size_t)dir * FX_NEDGES + eidx] = emf;
}

/* One CTA per (block, chunk of edge layers along i), one thread per node
 * (j, k) in [-1, 16]^2, marching along i.  A thread loads its cell (velocity,
 * field, density) and its three faces (two EMF products and the normal
 * velocity each) once per plane; values of the nodes j - 1 and k - 1 come through shared memory (two
 * buffers, one barrier per plane), values of plane i - 1 from its own
 * registers.  The cell EMFs are evaluated once per cell, as the reference's
 * per-cell grids are (src/prj_timeint.c:313-338); arithmetic of
 * prj_timeint_mhd_update_emf (src/prj_timeint.c:292-413).
 * Bound by memory latency and DRAM: 512 blocks 123 us, 528 MB at 4.3 TB/s
 * (compulsory about 475 MB), against 163 us and 729 MB for the kernel that
 * staged the cells of two layers and had each edge gather its eight face
 * values with the velocities in three-component tiles.  80 registers, 22
 * warps per SM; three CTAs per SM spill (177 us); loading one plane ahead
 * into registers spills, prefetching it into L2 or L1 measured 128-129 us.
 * The resistive term, zero in nearly every run, is a second pass, so that the
 * first carries nothing for it. */
constexpr int kEmfNodes = (FX_BS + 2) * (FX_BS + 2);
constexpr int kEmfThreads = (kEmfNodes + 31) / 32 * 32;

/* shared planes: cell EMFs, then what an edge reads from the node j - 1
 * (bv1 z, vr z, bv2 x, vr x) or k - 1 (bv2 y, vr y, bv1 x, vr x) */
enum { FX_EP_E1, FX_EP_E2, FX_EP_E3, FX_EP_BV1Z, FX_EP_VRZ, FX_EP_BV2X, FX_EP_VRX, FX_EP_BV2Y, FX_EP_VRY,
    FX_EP_BV1X, FX_EP_COUNT };

/* maximum artificial eta of an edge's four cells (src/prj_timeint.c:265-290) */
__device__ __noinline__ double fx_edge_eta(FxErr *err, const double *Wb, int b, int eidx, int c0, int su, int sr)
{
    const int cells[4] = {c0, c0 - su, c0 - su - sr, c0 - sr};
    double eta = 0.0;
    for (int n = 0; n < 4; ++n) {
        const double ce = fx_cell_eta(Wb[(size_t)FX_RHO * kPlane + cells[n]], Wb[(size_t)FX_YE * kPlane + cells[n]]);
        if (!isfinite(ce) || ce < 0.0) {
            fx_fail(err, FX_ERR_ETA, b, eidx);
        }
        if (ce > eta) {
            eta = ce;
        }
    }
    return eta;
}

/* two buffers of planes */
constexpr int kEmfSmem = 2 * FX_EP_COUNT * kEmfNodes * (int)sizeof(double);

/* curl B term of one edge, src/prj_mhd.c:682-709 */
__device__ __noinline__ double fx_edge_curl_b(const double *bf, const FxBlockDev &B, int bfslot, int dir, int i, int j, int k)
{
    const double *b1 = bf + (size_t)(0 * FX_NSTAGES + bfslot) * FX_NFACES;
    const double *b2 = bf + (size_t)(1 * FX_NSTAGES + bfslot) * FX_NFACES;
    const double *b3 = bf + (size_t)(2 * FX_NSTAGES + bfslot) * FX_NFACES;
    if (dir == 0) {
        return (b3[fx_face_idx(2, i, j, k)] - b3[fx_face_idx(2, i, j - 1, k)]) / B.dx[1] -
            (b2[fx_face_idx(1, i, j, k)] - b2[fx_face_idx(1, i, j, k - 1)]) / B.dx[2];
    }
    if (dir == 1) {
        return (b1[fx_face_idx(0, i, j, k)] - b1[fx_face_idx(0, i, j, k - 1)]) / B.dx[2] -
            (b3[fx_face_idx(2, i, j, k)] - b3[fx_face_idx(2, i - 1, j, k)]) / B.dx[0];
    }
    return (b2[fx_face_idx(1, i, j, k)] - b2[fx_face_idx(1, i - 1, j, k)]) / B.dx[0] -
        (b1[fx_face_idx(0, i, j, k)] - b1[fx_face_idx(0, i, j - 1, k)]) / B.dx[1];
}

/* infinite or NaN: the high word's exponent is all ones */
__device__ __forceinline__ bool fx_nonfinite(double x) { return (fx_hi(x) & 0x7ff00000) == 0x7ff00000; }

/* one edge from its four face EMFs, cell EMFs and normal velocities.  A
 * non-finite face EMF makes the sum of the four non-finite, so the result's
 * check covers it. */
template <int DIR>
__device__ __forceinline__ void fx_edge_store(const FxDev &D, int b, int i, int j, int k, const double (&f)[4],
    const double (&c)[4], const double (&vn)[4])
{
    const int eidx = fx_edge_idx(DIR, i, j, k);
    const double emf = fx_emf_upwind(f, c, vn);
    if (fx_nonfinite(emf) || fx_nonfinite(vn[0]) || fx_nonfinite(vn[1]) || fx_nonfinite(vn[2]) || fx_nonfinite(vn[3])) {
        fx_fail(D.err, FX_ERR_EMF_NONFINITE, b, eidx);
    }
    D.emf[(size_t)b * FX_EMF_COUNT + (size_t)DIR * FX_NEDGES + eidx] = emf;
}

/* the resistive term of one edge, added to the EMF its thread has stored */
__device__ __noinline__ void fx_edge_resist(const FxDev &D, int b, int wslot, int bfslot, int dir, int i, int j, int k)
{
    const int eidx = fx_edge_idx(dir, i, j, k);
    const double *Wb = D.W + (size_t)b * FX_W_COUNT(9) + (size_t)wslot * FX_NCELLS;
    const double eta = D.mhd_eta + fx_edge_eta(D.err, Wb, b, eidx, fx_lidx(i, j, k), fx_axis_stride((dir + 1) % 3),
        fx_axis_stride((dir + 2) % 3));
    if (eta == 0.0) {
        return;
    }
    double *e = D.emf + (size_t)b * FX_EMF_COUNT + (size_t)dir * FX_NEDGES + eidx;
    const double emf = *e + eta * fx_edge_curl_b(D.Bf + (size_t)b * FX_BF_COUNT, D.blk[b], bfslot, dir, i, j, k);
    if (!isfinite(emf)) {
        fx_fail(D.err, FX_ERR_EMF_NONFINITE, b, eidx);
    }
    *e = emf;
}

__global__ void __launch_bounds__(kEmfThreads, 2) k_emf(const __grid_constant__ FxDev D, const int *__restrict__ blist, int wslot,
    int bfslot, int nchunk)
{
    if (D.ctl->skip) {
        return;
    }
    extern __shared__ double emf_planes[]; /* [2][FX_EP_COUNT][kEmfNodes] */
    constexpr int ROW = FX_BS + 2;
    constexpr int N = kEmfNodes;
    const int b = blist[blockIdx.y];
    const int l0 = (FX_BS + 1) * (int)blockIdx.x / nchunk;
    const int l1 = (FX_BS + 1) * ((int)blockIdx.x + 1) / nchunk;
    const int t = threadIdx.x;
    const bool node = t < N;
    const int jj = t / ROW;
    const int j = jj - 1;
    const int k = t - jj * ROW - 1;
    const bool inner = node && j >= 0 && k >= 0; /* the node's edges exist */

    /* plane offset 0 is plane i = 0 */
    const int c0 = fx_lidx(0, node ? j : 0, node ? k : 0);
    constexpr int PL = FX_PBS * FX_PBS;
    const double *w = D.W + (size_t)b * FX_W_COUNT(9) + (size_t)wslot * FX_NCELLS + c0;
    const double *p1 = D.bv1 + (size_t)b * FX_BV_COUNT + c0;
    const double *p2 = D.bv2 + (size_t)b * FX_BV_COUNT + c0;
    const double *pv = D.vn + (size_t)b * FX_VN_COUNT + c0;

    /* values of plane i - 1 */
    double pE2 = 0.0, pE3 = 0.0, pE2k = 0.0, pE3j = 0.0, pbv1y = 0.0, pvry = 0.0, pbv2z = 0.0, pvrz = 0.0;
    bool resist = D.mhd_eta != 0.0;
    for (int i = l0 - 1; i < l1; ++i) {
        double *sp = emf_planes + (i & 1) * (FX_EP_COUNT * N) + t;
        double bv1y = 0.0, bv2z = 0.0;
        bool heavy = false;
        if (node) {
            const double *q = w + i * PL;
            const double rho = q[(size_t)FX_RHO * kPlane];
            const double v1 = q[(size_t)FX_V1 * kPlane], v2 = q[(size_t)FX_V2 * kPlane], v3 = q[(size_t)FX_V3 * kPlane];
            const double b1 = q[(size_t)FX_B1 * kPlane], b2 = q[(size_t)FX_B2 * kPlane], b3 = q[(size_t)FX_B3 * kPlane];
            double bv1x = 0.0, bv2x = 0.0, vrx = 0.0, bv2y = 0.0, vry = 0.0, bv1z = 0.0, vrz = 0.0;
            if (i >= 0) {
                bv1x = p1[i * PL];
                bv2x = p2[i * PL];
                vrx = pv[i * PL];
            }
            if (j >= 0) {
                bv1y = p1[FX_NCELLS + i * PL];
                bv2y = p2[FX_NCELLS + i * PL];
                vry = pv[FX_NCELLS + i * PL];
            }
            if (k >= 0) {
                bv1z = p1[2 * FX_NCELLS + i * PL];
                bv2z = p2[2 * FX_NCELLS + i * PL];
                vrz = pv[2 * FX_NCELLS + i * PL];
            }
            /* prj_timeint_mhd_cell_emf_all, src/prj_timeint.c:171-176 */
            const double E1 = b2 * v3 - b3 * v2;
            const double E2 = b3 * v1 - b1 * v3;
            const double E3 = b1 * v2 - b2 * v1;
            if (fx_nonfinite(E1) || fx_nonfinite(E2) || fx_nonfinite(E3)) {
                fx_fail(D.err, FX_ERR_EMF_NONFINITE, b, c0 + i * PL);
            }
            /* the artificial eta is zero up to this density (fx_cell_eta) */
            heavy = rho > FX_ETA_RHO_FLOOR;
            sp[FX_EP_E1 * N] = E1;
            sp[FX_EP_E2 * N] = E2;
            sp[FX_EP_E3 * N] = E3;
            sp[FX_EP_BV1Z * N] = bv1z;
            sp[FX_EP_VRZ * N] = vrz;
            sp[FX_EP_BV2X * N] = bv2x;
            sp[FX_EP_VRX * N] = vrx;
            sp[FX_EP_BV2Y * N] = bv2y;
            sp[FX_EP_VRY * N] = vry;
            sp[FX_EP_BV1X * N] = bv1x;
        }
        resist |= __syncthreads_or(heavy) != 0;
        if (!inner) {
            continue;
        }
        const double E2 = sp[FX_EP_E2 * N], E3 = sp[FX_EP_E3 * N];
        const double E2k = sp[FX_EP_E2 * N - 1], E3j = sp[FX_EP_E3 * N - ROW];
        const double vry = sp[FX_EP_VRY * N], vrz = sp[FX_EP_VRZ * N];
        if (i >= l0) {
            /* face0 = e (right-normal), face1 = e (up-normal), face2 = e - up
             * (right-normal), face3 = e - right (up-normal); cells e, e - up,
             * e - up - right, e - right */
            if (i < FX_BS) {
                const double f[4] = {sp[FX_EP_BV1Z * N], sp[FX_EP_BV2Y * N], sp[FX_EP_BV1Z * N - ROW], sp[FX_EP_BV2Y * N - 1]};
                const double c[4] = {sp[FX_EP_E1 * N], sp[FX_EP_E1 * N - ROW], sp[FX_EP_E1 * N - ROW - 1], sp[FX_EP_E1 * N - 1]};
                const double vn[4] = {vrz, vry, sp[FX_EP_VRZ * N - ROW], sp[FX_EP_VRY * N - 1]};
                fx_edge_store<0>(D, b, i, j, k, f, c, vn);
            }
            if (j < FX_BS) {
                const double f[4] = {sp[FX_EP_BV1X * N], bv2z, sp[FX_EP_BV1X * N - 1], pbv2z};
                const double c[4] = {E2, E2k, pE2k, pE2};
                const double vn[4] = {sp[FX_EP_VRX * N], vrz, sp[FX_EP_VRX * N - 1], pvrz};
                fx_edge_store<1>(D, b, i, j, k, f, c, vn);
            }
            if (k < FX_BS) {
                const double f[4] = {bv1y, sp[FX_EP_BV2X * N], pbv1y, sp[FX_EP_BV2X * N - ROW]};
                const double c[4] = {E3, pE3, pE3j, E3j};
                const double vn[4] = {vry, sp[FX_EP_VRX * N], pvry, sp[FX_EP_VRX * N - ROW]};
                fx_edge_store<2>(D, b, i, j, k, f, c, vn);
            }
        }
        pE2 = E2;
        pE3 = E3;
        pE2k = E2k;
        pE3j = E3j;
        pbv1y = bv1y;
        pvry = vry;
        pbv2z = bv2z;
        pvrz = vrz;
    }
    /* resistive edges (a run-time eta, or a cell above the density floor in
     * these planes) in a second pass, so that the pass above carries nothing
     * for them */
    if (resist && inner) {
        for (int i = l0; i < l1; ++i) {
            if (i < FX_BS) fx_edge_resist(D, b, wslot, bfslot, 0, i, j, k);
            if (j < FX_BS) fx_edge_resist(D, b, wslot, bfslot, 1, i, j, k);
            if (k < FX_BS) fx_edge_resist(D, b, wslot, bfslot, 2, i, j, k);
        }
    }
}

/* ------------------------------------------------------------------------ */
/* CT face update                                                            */
/* ------------------------------------------------------------------------ */
/* one face of direction DIR (compile-time, so the index arithmetic divides
 * by constants); grid (face chunk, direction, block) */
template <int DIR>
__device__ __forceinline__ void fx_bf_face(const FxDev &D, int b, int t, int stage, double dt)
{
    constexpr int x2 = DIR == 2 ? FX_BS + 1 : FX_BS;
    constexpr int x1 = DIR == 1 ? FX_BS + 1 : FX_BS;
    const int k = t % x2;
    t /= x2;
    const int j = t % x1;
    const int i = t / x1;
    const int src_slot = stage == 2 ? 1 : 0;
    const int dst_slot = stage == 1 ? 1 : 0;
    double *bf = D.Bf + (size_t)b * FX_BF_COUNT;
    const double *e = D.emf + (size_t)b * FX_EMF_COUNT;
    const double *e1 = e;
    const double *e2 = e + FX_NEDGES;
    const double *e3 = e + 2 * FX_NEDGES;
    const FxBlockDev &B = D.blk[b];
    const int f = fx_face_idx(DIR, i, j, k);
    double value = bf[((size_t)DIR * FX_NSTAGES + src_slot) * FX_NFACES + f];
    if (DIR == 0) {
        value += -dt * (e3[fx_edge_idx(2, i, j + 1, k)] - e3[fx_edge_idx(2, i, j, k)]) / B.dx[1];
        value += dt * (e2[fx_edge_idx(1, i, j, k + 1)] - e2[fx_edge_idx(1, i, j, k)]) / B.dx[2];
    } else if (DIR == 1) {
        value += -dt * (e1[fx_edge_idx(0, i, j, k + 1)] - e1[fx_edge_idx(0, i, j, k)]) / B.dx[2];
        value += dt * (e3[fx_edge_idx(2, i + 1, j, k)] - e3[fx_edge_idx(2, i, j, k)]) / B.dx[0];
    } else {
        value += -dt * (e2[fx_edge_idx(1, i + 1, j, k)] - e2[fx_edge_idx(1, i, j, k)]) / B.dx[0];
        value += dt * (e1[fx_edge_idx(0, i, j + 1, k)] - e1[fx_edge_idx(0, i, j, k)]) / B.dx[1];
    }
    if (!isfinite(value)) {
        fx_fail(D.err, FX_ERR_BF_NONFINITE, b, f);
    }
    if (stage == 2) {
        value = 0.5 * bf[((size_t)DIR * FX_NSTAGES + 0) * FX_NFACES + f] + 0.5 * value;
    }
    bf[((size_t)DIR * FX_NSTAGES + dst_slot) * FX_NFACES + f] = value;
}

__global__ void __launch_bounds__(128) k_bf_update(FxDev D, const int *__restrict__ blist, int stage)
{
    if (D.ctl->skip) {
        return;
    }
    constexpr int NF = (FX_BS + 1) * FX_BS * FX_BS;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= NF) {
        return;
    }
    const double dt = D.ctl->dt_stage;
    const int b = blist[blockIdx.z];
    switch (blockIdx.y) {
    case 0: fx_bf_face<0>(D, b, t, stage, dt); break;
    case 1: fx_bf_face<1>(D, b, t, stage, dt); break;
    default: fx_bf_face<2>(D, b, t, stage, dt); break;
    }
}

/* ------------------------------------------------------------------------ */
/* Cell update (flux divergence + sources + RK2 combine + cons2prim)         */
/* ------------------------------------------------------------------------ */
/* a cell's timestep, prj_timeint_calc_dt (src/prj_timeint.c:2144-2256) */
__device__ __forceinline__ double fx_cell_dt(double cfl, double g, double rho, double eint, double v1, double v2,
    double v3, const FxBlockDev &B)
{
    const double p = fx_pressure(g, rho, eint);
    const double cs = sqrt(g * p / rho);
    const double denom = (fabs(v1) + cs) / B.dx[0] + (fabs(v2) + cs) / B.dx[1] + (fabs(v3) + cs) / B.dx[2];
    return cfl / denom;
}

/* STAGE 1 / 2: the RK2 stages; STAGE 0: the stage-1 arithmetic written in
 * place to slot 0 with the field of Bf slot 0 (an eSSPRK substep,
 * prj_timeint_eSSPRK_step, src/prj_timeint.c:2484-2508).
 * FULL: the plain form (rhs stored), else the batched one.
 * DT (the RK2 driver loop): the new state's timestep minimum goes to D.red[0]
 * for the next step, which then needs no pass over the state for it (the ghost
 * fill leaves active cells alone): a step of 8 blocks 68.1 -> 65.1 us, of 512
 * blocks 2025 -> 1983. */
template <bool MHD, int STAGE, bool FULL, bool DT = false>
__global__ void __launch_bounds__(128) k_cell_update(FxDev D, const int *__restrict__ blist, int gravity)
{
    if (D.ctl->skip) {
        return;
    }
    const double dt = D.ctl->dt_stage;
    const int b = blist[blockIdx.y];
    constexpr int nv = MHD ? 9 : 6;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= FX_BS * FX_BS * FX_BS) {
        return;
    }
    const int k = t % FX_BS;
    const int j = (t / FX_BS) % FX_BS;
    const int i = t / (FX_BS * FX_BS);
    const int c = fx_lidx(i, j, k);
    const FxBlockDev &B = D.blk[b];
    const double *W = D.W + (size_t)b * FX_W_COUNT(nv);

    /* prj_flux_div, src/prj_flux.c:2523-2533 (hydro components; the B
     * components are replaced by the face average below) */
    double fluxdiv[6];
#pragma unroll
    for (int v = 0; v < 6; ++v) {
        double f[3][2];
        const double *cf = D.cf + (size_t)b * FX_CF_COUNT;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double *q = cf + v * fx_cf_plane(d) + fx_cf_idx(d, i, j, k);
            f[d][0] = q[0];
            f[d][1] = q[d == 0 ? FX_BS * FX_BS : d == 1 ? FX_BS : 1];
        }
        fluxdiv[v] = -(B.area[0] * (f[0][1] - f[0][0]) + B.area[1] * (f[1][1] - f[1][0]) +
            B.area[2] * (f[2][1] - f[2][0])) / B.vol;
    }

    double w[9];
    double u[9];
#pragma unroll
    for (int v = 0; v < nv; ++v) {
        w[v] = W[(size_t)v * kPlane + c];
    }
    fx_prim2cons<MHD>(w, u);

    /* source terms: rhs = 0, then the static-gravity terms of
     * prj_src_monopole_gravity with the stage primitives (src/prj_src.c:32-139) */
    double rhs[6];
#pragma unroll
    for (int v = 0; v < 6; ++v) {
        rhs[v] = 0.0;
    }
    if (gravity) {
        const double *Ws = W + (size_t)(STAGE == 2 ? 1 : 0) * FX_NCELLS;
        const double *g = D.grav + (size_t)b * FX_GRAV_COUNT;
        const double g1 = g[c];
        const double g2 = g[FX_NCELLS + c];
        const double g3 = g[2 * FX_NCELLS + c];
        const double rho = Ws[(size_t)FX_RHO * kPlane + c];
        rhs[FX_V1] += rho * g1;
        rhs[FX_V2] += rho * g2;
        rhs[FX_V3] += rho * g3;
        double vf[3][2];
        const double *vn = D.vn + (size_t)b * FX_VN_COUNT + c;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            vf[d][0] = vn[d * FX_NCELLS];
            vf[d][1] = vn[d * FX_NCELLS + fx_axis_stride(d)];
        }
        const double v_avg1 = (vf[0][0] + vf[0][1]) * 0.5;
        const double v_avg2 = (vf[1][0] + vf[1][1]) * 0.5;
        const double v_avg3 = (vf[2][0] + vf[2][1]) * 0.5;
        rhs[FX_ETOT] += rho * (v_avg1 * g1 + v_avg2 * g2 + v_avg3 * g3);
    }
    if constexpr (FULL) {
        double *r = D.rhs + (size_t)b * FX_RHS_COUNT(nv);
#pragma unroll
        for (int v = 0; v < nv; ++v) {
            r[fx_bidx(nv, v, i, j, k)] = v < 6 ? rhs[v] : 0.0;
        }
    }

    /* dt_src from the start-of-step total energy,
     * prj_timeint_update_dt_src_values (src/prj_timeint.c:533-565) */
    const double dt_src = 0.02 * u[FX_ETOT] / (fabs(rhs[FX_ETOT]) + 1.0e-50);

    double un[9];
    if (STAGE != 2) {
#pragma unroll
        for (int v = 0; v < 6; ++v) {
            un[v] = u[v] + dt * (rhs[v] + fluxdiv[v]);
        }
    } else {
        double w1[9];
        double u1[9];
        const double *W1 = W + FX_NCELLS;
#pragma unroll
        for (int v = 0; v < nv; ++v) {
            w1[v] = W1[(size_t)v * kPlane + c];
        }
        fx_prim2cons<MHD>(w1, u1);
#pragma unroll
        for (int v = 0; v < 6; ++v) {
            const double u_trial = u1[v] + dt * (rhs[v] + fluxdiv[v]);
            un[v] = 0.5 * u[v] + 0.5 * u_trial;
        }
    }
    if (MHD) {
        /* cell B from the updated faces, src/prj_timeint.c:498-510 */
        const int bslot = STAGE == 1 ? 1 : 0;  /* slot the CT update wrote */
        const double *bf = D.Bf + (size_t)b * FX_BF_COUNT;
        const double *b1 = bf + (size_t)(0 * FX_NSTAGES + bslot) * FX_NFACES;
        const double *b2 = bf + (size_t)(1 * FX_NSTAGES + bslot) * FX_NFACES;
        const double *b3 = bf + (size_t)(2 * FX_NSTAGES + bslot) * FX_NFACES;
        un[FX_B1] = 0.5 * (b1[fx_face_idx(0, i, j, k)] + b1[fx_face_idx(0, i + 1, j, k)]);
        un[FX_B2] = 0.5 * (b2[fx_face_idx(1, i, j, k)] + b2[fx_face_idx(1, i, j + 1, k)]);
        un[FX_B3] = 0.5 * (b3[fx_face_idx(2, i, j, k)] + b3[fx_face_idx(2, i, j, k + 1)]);
        if (!isfinite(un[FX_B1]) || !isfinite(un[FX_B2]) || !isfinite(un[FX_B3])) {
            fx_fail(D.err, FX_ERR_B_NONFINITE, b, c);
        }
    }
    double wn[9];
    fx_cons2prim<MHD>(un, wn);
    double *Wd = D.W + (size_t)b * FX_W_COUNT(nv) + (size_t)(STAGE == 1 ? 1 : 0) * FX_NCELLS;
#pragma unroll
    for (int v = 0; v < nv; ++v) {
        Wd[(size_t)v * kPlane + c] = wn[v];
    }

    /* block-wide minimum of dt_src (and of the timestep), then one atomic per CTA */
    constexpr int NK = DT ? 2 : 1;
    __shared__ unsigned long long smin[NK][4];
    unsigned long long key[NK];
    key[0] = fx_double_key(dt_src);
    if (dt_src != dt_src) {
        key[0] = ~0ULL;
    }
    if constexpr (DT) {
        const double dt_cell = fx_cell_dt(D.ctl->cfl, D.gamma, wn[FX_RHO], wn[FX_EINT], wn[FX_V1], wn[FX_V2], wn[FX_V3], B);
        key[1] = dt_cell == dt_cell ? fx_double_key(dt_cell) : ~0ULL;
    }
#pragma unroll
    for (int n = 0; n < NK; ++n) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const unsigned long long o = __shfl_down_sync(0xffffffffu, key[n], off);
            key[n] = o < key[n] ? o : key[n];
        }
        if ((threadIdx.x & 31) == 0) {
            smin[n][threadIdx.x >> 5] = key[n];
        }
    }
    __syncthreads();
    if (threadIdx.x < NK) {
        const int n = threadIdx.x;
        unsigned long long m = smin[n][0];
        for (int q = 1; q < (int)(blockDim.x >> 5); ++q) {
            m = smin[n][q] < m ? smin[n][q] : m;
        }
        atomicMin(&D.red[1 - n], m);
    }
}

/* ------------------------------------------------------------------------ */
/* EOS fill (eosvar = p, T, gamma from the stage primitives)                 */
/* ------------------------------------------------------------------------ */
__global__ void k_eos_fill(FxDev D, const int *__restrict__ blist, int wslot, int active_only)
{
    if (D.ctl->skip) {
        return;
    }
    const int b = blist[blockIdx.y];
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    int i, j, k;
    if (active_only) {
        if (t >= FX_BS * FX_BS * FX_BS) return;
        k = t % FX_BS;
        j = (t / FX_BS) % FX_BS;
        i = t / (FX_BS * FX_BS);
    } else {
        if (t >= FX_NCELLS) return;
        k = t % FX_PBS - FX_NG;
        j = (t / FX_PBS) % FX_PBS - FX_NG;
        i = t / (FX_PBS * FX_PBS) - FX_NG;
    }
    const int c = fx_lidx(i, j, k);
    const double *W = D.W + (size_t)b * FX_W_COUNT(D.nv) + (size_t)wslot * FX_NCELLS;
    const double rho = W[(size_t)FX_RHO * kPlane + c];
    const double eint = W[(size_t)FX_EINT * kPlane + c];
    if (rho == 0.0) {
        fx_fail(D.err, FX_ERR_EOS_ZERO_RHO, b, c);
    }
    const double g = D.gamma;
    double *e = D.eos + (size_t)b * FX_EOS_COUNT;
    e[fx_bidx(3, FX_EOS_P, i, j, k)] = fx_pressure(g, rho, eint);
    e[fx_bidx(3, FX_EOS_T, i, j, k)] = fx_temperature(g, eint);
    e[fx_bidx(3, FX_EOS_G, i, j, k)] = g;
}

/* ------------------------------------------------------------------------ */
/* dt = min over active cells of cfl / sum_d (|v_d| + c_s) / dx_d            */
/* ------------------------------------------------------------------------ */
__global__ void __launch_bounds__(256) k_calc_dt(FxDev D, const int *__restrict__ blist, int wslot, double cfl)
{
    const int b = blist[blockIdx.y];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    unsigned long long key = ~0ULL;
    if (t < FX_BS * FX_BS * FX_BS) {
        const int k = t % FX_BS;
        const int j = (t / FX_BS) % FX_BS;
        const int i = t / (FX_BS * FX_BS);
        const int c = fx_lidx(i, j, k);
        const double *W = D.W + (size_t)b * FX_W_COUNT(D.nv) + (size_t)wslot * FX_NCELLS;
        const FxBlockDev &B = D.blk[b];
        const double dt_cell = fx_cell_dt(cfl, D.gamma, W[(size_t)FX_RHO * kPlane + c], W[(size_t)FX_EINT * kPlane + c],
            W[(size_t)FX_V1 * kPlane + c], W[(size_t)FX_V2 * kPlane + c], W[(size_t)FX_V3 * kPlane + c], B);
        if (dt_cell == dt_cell) {
            key = fx_double_key(dt_cell);
        }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const unsigned long long o = __shfl_down_sync(0xffffffffu, key, off);
        key = o < key ? o : key;
    }
    __shared__ unsigned long long smin[8];
    if ((threadIdx.x & 31) == 0) {
        smin[threadIdx.x >> 5] = key;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long m = smin[0];
        for (int q = 1; q < (int)(blockDim.x >> 5); ++q) {
            m = smin[q] < m ? smin[q] : m;
        }
        atomicMin(&D.red[0], m);
    }
}

__global__ void k_reset_reductions(FxDev D, int which)
{
    /* initial values of the reference's reductions: dt_min = 1e99
     * (src/prj_timeint.c:2147), dt_src = 1e100 (src/main.c:491) */
    if (which & 1) D.red[0] = fx_double_key(1.0e99);
    if (which & 2) D.red[1] = fx_double_key(1.0e100);
}

__device__ __forceinline__ double fx_key_double(unsigned long long key)
{
    const unsigned long long bits = (key >> 63) ? (key & 0x7fffffffffffffffULL) : ~key;
    return __longlong_as_double((long long)bits);
}

/* dt selection of the driver loop, src/main.c:485-517 (no output events) */
__global__ void k_step_begin(FxDev D)
{
    FxCtl *c = D.ctl;
    if (!(c->time < c->t_end)) {
        c->skip = 1;
        return;
    }
    c->skip = 0;
    /* prj_timeint_calc_dt's minimum, times 6 for eSSPRK10_4 */
    const double dt_new = fx_key_double(D.red[0]) * c->dt_mult;
    D.red[0] = fx_double_key(1.0e99); /* the next minimum starts afresh */
    if (c->dt_prev > 0.0) {
        const double dt_limit = c->dt_factor * c->dt_prev;
        c->dt_prev = dt_new <= dt_limit ? dt_new : dt_limit;
    } else {
        c->dt_prev = dt_new;
    }
    double dt_step = c->dt_prev;
    if (c->time + dt_step > c->t_end) {
        dt_step = c->t_end - c->time;
    }
    c->dt = dt_step;
    c->dt_stage = dt_step;
    D.red[1] = fx_double_key(1.0e100);
}

/* after the step: dt_src clamp and time advance, src/main.c:555-562 */
__global__ void k_step_end(FxDev D)
{
    FxCtl *c = D.ctl;
    if (c->skip) {
        return;
    }
    const double dt_src = fx_key_double(D.red[1]);
    c->dt_src = dt_src;
    if (c->cfl * dt_src < c->dt_prev) {
        c->dt_prev = c->cfl * dt_src;
    }
    c->time += c->dt;
    c->step += 1;
}

/* ------------------------------------------------------------------------ */
/* Ghost-fill programs                                                       */
/* ------------------------------------------------------------------------ */

/* the primitives the fill writes: all but the cell-centred field, which
 * follows from the faces */
constexpr int kGhostVars = 6;

/* prj_reconstruct_cell_for_prolongate_minmod (src/prj_reconstruct.h:111-143):
 * per axis base + slope * target, combined as vx + vy + vz - 2 base; target
 * offsets are +-1/4 of a coarse cell.  use_BJ = 1 takes fx_bj_cell /
 * fx_bj_face on the full 27-cell (3x3-face) stencil instead. */
__device__ __forceinline__ double fx_prolong_cell(const double *q, int c, double tx, double ty, double tz)
{
    const double base = q[c];
    const double vx = base + fx_minmod_slope(q[c - FX_PBS * FX_PBS], base, q[c + FX_PBS * FX_PBS]) * tx;
    const double vy = base + fx_minmod_slope(q[c - FX_PBS], base, q[c + FX_PBS]) * ty;
    const double vz = base + fx_minmod_slope(q[c - 1], base, q[c + 1]) * tz;
    return vx + vy + vz - 2.0 * base;
}

/* prj_reconstruct_face_for_prolongate_minmod (src/prj_reconstruct.h:222-246)
 * on the face stencil of direction d about face f: tangential axes t0 < t1
 * with face-index strides s0, s1 */
__device__ __forceinline__ double fx_prolong_face(const double *q, int f, int s0, int s1, double t0, double t1)
{
    const double base = q[f];
    const double vx = base + fx_minmod_slope(q[f - s0], base, q[f + s0]) * t0;
    const double vy = base + fx_minmod_slope(q[f - s1], base, q[f + s1]) * t1;
    return vx + vy - base;
}

/* BJ: the program may hold Barth-Jespersen prolongations (use_BJ); the
 * other instance keeps the copy-dominated wave kernel at its small register
 * count */
template <bool BJ>
__device__ __forceinline__ void fx_ghost_cell_op(const FxDev &D, const FxGop op, int wslot)
{
    const int db = FX_CELL_BLOCK(op.dst);
    const int dc = FX_CELL_IDX(op.dst);
    const int sb = FX_CELL_BLOCK(op.src);
    const int sc = FX_CELL_IDX(op.src);
    double *Wd = D.W + (size_t)db * FX_W_COUNT(D.nv) + (size_t)wslot * FX_NCELLS;
    const double *Ws = D.W + (size_t)sb * FX_W_COUNT(D.nv) + (size_t)wslot * FX_NCELLS;
    if constexpr (BJ) {
        if (op.type == FX_GOP_PROLONG_BJ) {
            const double tx = (op.aux & 4) ? 0.25 : -0.25;
            const double ty = (op.aux & 2) ? 0.25 : -0.25;
            const double tz = (op.aux & 1) ? 0.25 : -0.25;
#pragma unroll 1
            for (int v = 0; v < kGhostVars; ++v) {
                const double *q = Ws + (size_t)v * kPlane + sc;
                Wd[(size_t)v * kPlane + dc] = fx_bj_cell(
                    [q](int di, int dj, int dk) { return q[(di * FX_PBS + dj) * FX_PBS + dk]; }, tx, ty, tz);
            }
            return;
        }
    }
    /* every variable's value first, then the stores: the loads of all
     * variables are in flight together (the wave's operations are conflict
     * free, so no store of the wave feeds a load of it) */
    double val[kGhostVars];
    switch (op.type) {
    case FX_GOP_COPY:
    case FX_GOP_COPY_NEG:
    case FX_GOP_COPY_USER:
#pragma unroll
        for (int v = 0; v < kGhostVars; ++v) {
            val[v] = Ws[(size_t)v * kPlane + sc];
        }
        if (op.type == FX_GOP_COPY_NEG) {
#pragma unroll
            for (int v = 0; v < kGhostVars; ++v) {
                if (v == op.aux) val[v] = -val[v];
            }
        } else if (op.type == FX_GOP_COPY_USER && op.aux) {
            val[FX_V1] = 5.0;
        }
        break;
    case FX_GOP_RESTRICT:
#pragma unroll
        for (int v = 0; v < kGhostVars; ++v) {
            const double *q = Ws + (size_t)v * kPlane + sc;
            /* order of src/prj_boundary.c:238-261 */
            val[v] = 0.125 *
                (q[0] + q[1] + q[FX_PBS] + q[FX_PBS + 1] +
                 q[FX_PBS * FX_PBS] + q[FX_PBS * FX_PBS + 1] +
                 q[FX_PBS * FX_PBS + FX_PBS] + q[FX_PBS * FX_PBS + FX_PBS + 1]);
        }
        break;
    case FX_GOP_PROLONG: {
        /* target offsets of src/prj_boundary.c:318-320 */
        const double tx = (op.aux & 4) ? 0.25 : -0.25;
        const double ty = (op.aux & 2) ? 0.25 : -0.25;
        const double tz = (op.aux & 1) ? 0.25 : -0.25;
#pragma unroll
        for (int v = 0; v < kGhostVars; ++v) {
            val[v] = fx_prolong_cell(Ws + (size_t)v * kPlane, sc, tx, ty, tz);
        }
        break;
    }
    default:
        return;
    }
#pragma unroll
    for (int v = 0; v < kGhostVars; ++v) {
        Wd[(size_t)v * kPlane + dc] = val[v];
    }
}

__device__ __forceinline__ int fx_face_key_block(int key) { return key >> 15; }
__device__ __forceinline__ int fx_face_key_idx(int key) { return key & 32767; }

/* the value of one face operation (its loads) and where it goes; the store
 * is left to the caller, so that a thread can issue the loads of several
 * operations before their stores (the operations of a wave are conflict
 * free).  Null for an unknown type. */
__device__ __forceinline__ double *fx_ghost_face_value(const FxDev &D, const FxGop op, int bfslot, double &v)
{
    const int dir = op.aux & 3;
    const int db = fx_face_key_block(op.dst);
    const int df = fx_face_key_idx(op.dst);
    const int sb = fx_face_key_block(op.src);
    const int sf = fx_face_key_idx(op.src);
    double *Bd = D.Bf + (size_t)db * FX_BF_COUNT + ((size_t)dir * FX_NSTAGES + bfslot) * FX_NFACES;
    const double *Bs = D.Bf + (size_t)sb * FX_BF_COUNT + ((size_t)dir * FX_NSTAGES + bfslot) * FX_NFACES;
    if (op.type == FX_FOP_COPY) {
        v = Bs[sf];
        return Bd + df;
    }
    if (op.type == FX_FOP_RESTRICT) {
        /* 0.25*(s0 + s0+t1 + s0+t0 + s0+t0+t1), src/prj_boundary.c:738-764 */
        const int o1 = (op.aux >> 2) & 1023;   /* stride of tan1 */
        const int o0 = (op.aux >> 12) & 1023;  /* stride of tan0 */
        v = 0.25 * (Bs[sf] + Bs[sf + o1] + Bs[sf + o0] + Bs[sf + o0 + o1]);
        return Bd + df;
    }
    return nullptr;
}

/* face operations per thread of the wave kernel: a face copy moves one
 * double, so one operation per thread leaves too few loads in flight to
 * keep HBM busy */
constexpr int FX_GW_FACE_OPS = 4;

/* face-index offset of a unit step along axis a for faces of direction d */
__device__ __forceinline__ int fx_face_stride(int d, int a)
{
    return fx_face_idx(d, a == 0, a == 1, a == 2) - fx_face_idx(d, 0, 0, 0);
}

/* One Toth-Roe group: prj_mhd_prolong_bf_from_buffer (src/prj_mhd.c:374-512)
 * with prj_mhd_compute_buffer_inner_fluxes (src/prj_mhd.c:309-372), in the
 * reference's operation order.  Outer faces are area-weighted fluxes; kept
 * faces contribute their current fine value.
 * Four neighbouring lanes share a group, lane 2 a + b taking the sub-faces
 * (a, b): six outer and three inner faces each, where one thread had 24 and
 * 12 one after the other, and of the six sums over the outer fluxes (eight
 * divisions in three of them) the lanes 0 to 2 one pair each.  The fluxes and
 * sums go from lane to lane by shuffles, so every lane of the warp comes here;
 * `live` lanes store.  Latency bound: a fill's later waves have few groups.
 * 470-block blast: a fill of seven waves 288 -> 234 us. */
__device__ __forceinline__ void fx_ghost_prolong_group(const FxDev &D, const FxPop &op, int slot, bool live)
{
    const int lane = threadIdx.x & 3;
    const int a = lane >> 1, b = lane & 1;
    const double sa = a ? 1.0 : -1.0, sb = b ? 1.0 : -1.0;
    const int f0[3] = {(op.pos & 31) - FX_NG, ((op.pos >> 5) & 31) - FX_NG, ((op.pos >> 10) & 31) - FX_NG};
    const int c0[3] = {((op.pos >> 15) & 31) - FX_NG, ((op.pos >> 20) & 31) - FX_NG, ((op.pos >> 25) & 31) - FX_NG};
    const FxBlockDev &fb = D.blk[op.fine];
    const double area[3] = {fb.dx[1] * fb.dx[2], fb.dx[0] * fb.dx[2], fb.dx[0] * fb.dx[1]};
    /* this lane's outer fluxes [d][side] */
    double of[3][2];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int t0 = d == 0 ? 1 : 0;
        const int t1 = d == 2 ? 1 : 2;
        double *Bfine = D.Bf + (size_t)op.fine * FX_BF_COUNT + ((size_t)d * FX_NSTAGES + slot) * FX_NFACES;
        const double *Bc = D.Bf + (size_t)op.coarse * FX_BF_COUNT + ((size_t)d * FX_NSTAGES + slot) * FX_NFACES;
        const int s0 = fx_face_stride(d, t0);
        const int s1 = fx_face_stride(d, t1);
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            int y[3] = {c0[0], c0[1], c0[2]};
            y[d] += side;
            const int cf = fx_face_idx(d, y[0], y[1], y[2]);
            const int q = 8 * d + 4 * side + lane;
            int x[3] = {f0[0], f0[1], f0[2]};
            x[d] += 2 * side;
            x[t0] += a;
            x[t1] += b;
            const int xf = fx_face_idx(d, x[0], x[1], x[2]);
            if ((op.keep >> q) & 1) {
                of[d][side] = Bfine[xf] * area[d];
            } else {
                const double ta = a ? 0.25 : -0.25;
                const double tb = b ? 0.25 : -0.25;
                const double *qc = Bc + cf;
                const double value = (op.flags & 1)
                    ? fx_bj_face([qc, s0, s1](int d0, int d1) { return qc[d0 * s0 + d1 * s1]; }, ta, tb)
                    : fx_prolong_face(Bc, cf, s0, s1, ta, tb);
                const double flux = value * area[d];
                of[d][side] = flux;
                if (live && ((op.owrite >> q) & 1)) {
                    Bfine[xf] = flux / area[d];
                }
            }
        }
    }
    /* u[i][j][k] of the reference: u[0|2][j][k] is the outer flux of direction
     * 0 on side 0|1 at sub-face (j, k), v[i][0|2][k] of direction 1 at (i, k),
     * w[i][j][0|2] of direction 2 at (i, j).  Lane n sums, over i, j, k in
     * this order, for n = 0, 1, 2:
     *   Uxx += si sj v + si sk w, Vyy += sj sk w + sj si u, Wzz += sk si u + sk sj v
     *   Uxyz += si sj sk u / (dx2s + dx3s), and cyclically
     * (products of signs are exact) */
    const double dx1s = fb.dx[0] * fb.dx[0];
    const double dx2s = fb.dx[1] * fb.dx[1];
    const double dx3s = fb.dx[2] * fb.dx[2];
    const int n = lane < 3 ? lane : 0;
    const double den = n == 0 ? dx2s + dx3s : n == 1 ? dx1s + dx3s : dx1s + dx2s;
    double S = 0.0, T = 0.0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double si = i ? 1.0 : -1.0;
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const double sj = j ? 1.0 : -1.0;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const double sk = k ? 1.0 : -1.0;
                const int quad = threadIdx.x & 28;
                const double u = __shfl_sync(0xffffffffu, of[0][i], quad | (2 * j + k));
                const double v = __shfl_sync(0xffffffffu, of[1][j], quad | (2 * i + k));
                const double w = __shfl_sync(0xffffffffu, of[2][k], quad | (2 * i + j));
                const double X = n == 0 ? si * sj * v : n == 1 ? sj * sk * w : sk * si * u;
                const double Y = n == 0 ? si * sk * w : n == 1 ? sj * si * u : sk * sj * v;
                S += X + Y;
                T += si * sj * sk * (n == 0 ? u : n == 1 ? v : w) / den;
            }
        }
    }
    S *= 0.125;
    T *= 0.125;
    const int quad = threadIdx.x & 28;
    const double Uxx = __shfl_sync(0xffffffffu, S, quad);
    const double Vyy = __shfl_sync(0xffffffffu, S, quad | 1);
    const double Wzz = __shfl_sync(0xffffffffu, S, quad | 2);
    const double Uxyz = __shfl_sync(0xffffffffu, T, quad);
    const double Vxyz = __shfl_sync(0xffffffffu, T, quad | 1);
    const double Wxyz = __shfl_sync(0xffffffffu, T, quad | 2);
    if (!live) {
        return;
    }
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int t0 = d == 0 ? 1 : 0;
        const int t1 = d == 2 ? 1 : 2;
        if (!((op.iwrite >> (4 * d + lane)) & 1)) continue;
        double flux;
        if (d == 0) {        /* u[1][j][k], (a, b) = (j, k) */
            flux = 0.5 * (of[0][1] + of[0][0]) + Uxx + sb * dx3s * Vxyz + sa * dx2s * Wxyz;
        } else if (d == 1) { /* v[i][1][k], (a, b) = (i, k) */
            flux = 0.5 * (of[1][1] + of[1][0]) + Vyy + sa * dx1s * Wxyz + sb * dx3s * Uxyz;
        } else {             /* w[i][j][1], (a, b) = (i, j) */
            flux = 0.5 * (of[2][1] + of[2][0]) + Wzz + sb * dx2s * Uxyz + sa * dx1s * Vxyz;
        }
        const double value = flux / area[d];
        int x[3] = {f0[0], f0[1], f0[2]};
        x[d] += 1;
        x[t0] += a;
        x[t1] += b;
        const int xf = fx_face_idx(d, x[0], x[1], x[2]);
        if (!isfinite(value)) {
            fx_fail(D.err, FX_ERR_BF_NONFINITE, op.fine, xf);
        }
        D.Bf[(size_t)op.fine * FX_BF_COUNT + ((size_t)d * FX_NSTAGES + slot) * FX_NFACES + xf] = value;
    }
}

/* cell-centred field of one cell from its faces: prj_mhd_bf2bc_impl
 * (src/prj_mhd.c:555-603).  The metric factor sqrt(gamma) is 1 outside
 * dynamical GR; the reference's division by it is exact and omitted. */
__device__ __forceinline__ void fx_ghost_b_op(const FxDev &D, const FxBop op, int slot)
{
    double v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int k0 = op.f[2 * d];
        const int k1 = op.f[2 * d + 1];
        const double *b0 = D.Bf + (size_t)fx_face_key_block(k0) * FX_BF_COUNT +
            ((size_t)d * FX_NSTAGES + slot) * FX_NFACES;
        const double *b1 = D.Bf + (size_t)fx_face_key_block(k1) * FX_BF_COUNT +
            ((size_t)d * FX_NSTAGES + slot) * FX_NFACES;
        v[d] = 0.5 * (b0[fx_face_key_idx(k0)] + b1[fx_face_key_idx(k1)]);
    }
    const int b = FX_CELL_BLOCK(op.dst);
    const int c = FX_CELL_IDX(op.dst);
    if (!isfinite(v[0]) || !isfinite(v[1]) || !isfinite(v[2])) {
        fx_fail(D.err, FX_ERR_B_NONFINITE, b, c);
    }
    double *W = D.W + (size_t)b * FX_W_COUNT(9) + (size_t)slot * FX_NCELLS;
    W[(size_t)FX_B1 * kPlane + c] = v[0];
    W[(size_t)FX_B2 * kPlane + c] = v[1];
    W[(size_t)FX_B3 * kPlane + c] = v[2];
}

/* two neighbouring doubles: one 16-byte access where the index is even (the
 * block arrays and their planes start 16-byte aligned), else two */
__device__ __forceinline__ double2 fx_load2(const double *p, int i)
{
    if ((i & 1) == 0) return *reinterpret_cast<const double2 *>(p + i);
    return make_double2(p[i], p[i + 1]);
}

__device__ __forceinline__ void fx_store2(double *p, int i, double2 v)
{
    if ((i & 1) == 0) {
        *reinterpret_cast<double2 *>(p + i) = v;
    } else {
        p[i] = v.x;
        p[i + 1] = v.y;
    }
}

/* one or two neighbouring cell copies, every load ahead of the stores */
__device__ __forceinline__ void fx_ghost_cell_copy(const FxDev &D, const FxPair op, int slot)
{
    const int dst = op.dst & 0x7fffffff;
    const int sc = FX_CELL_IDX(op.src), dc = FX_CELL_IDX(dst);
    const double *Ws = D.W + (size_t)FX_CELL_BLOCK(op.src) * FX_W_COUNT(D.nv) + (size_t)slot * FX_NCELLS;
    double *Wd = D.W + (size_t)FX_CELL_BLOCK(dst) * FX_W_COUNT(D.nv) + (size_t)slot * FX_NCELLS;
    if (op.dst < 0) {
        double val[kGhostVars];
#pragma unroll
        for (int v = 0; v < kGhostVars; ++v) val[v] = Ws[(size_t)v * kPlane + sc];
#pragma unroll
        for (int v = 0; v < kGhostVars; ++v) Wd[(size_t)v * kPlane + dc] = val[v];
        return;
    }
    double2 val[kGhostVars];
#pragma unroll
    for (int v = 0; v < kGhostVars; ++v) val[v] = fx_load2(Ws + (size_t)v * kPlane, sc);
#pragma unroll
    for (int v = 0; v < kGhostVars; ++v) fx_store2(Wd + (size_t)v * kPlane, dc, val[v]);
}

/* direction array of a pair's face key, and the face in it */
__device__ __forceinline__ double *fx_pair_faces(const FxDev &D, int key, int slot, int &f)
{
    const unsigned bd = ((unsigned)key & 0x7fffffffu) >> 14;
    f = key & 16383;
    /* block b, direction d: (2 (3 b + d) + slot) faces in */
    return D.Bf + ((size_t)bd * FX_NSTAGES + slot) * FX_NFACES;
}

/* cell-centred field of two neighbouring cells (fx_ghost_b_op) */
__device__ __forceinline__ void fx_ghost_b_pair(const FxDev &D, const FxBop op, int slot)
{
    double2 v[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int k0 = op.f[2 * d];
        const int k1 = op.f[2 * d + 1];
        const double2 a = fx_load2(D.Bf + (size_t)fx_face_key_block(k0) * FX_BF_COUNT +
            ((size_t)d * FX_NSTAGES + slot) * FX_NFACES, fx_face_key_idx(k0));
        const double2 b = fx_load2(D.Bf + (size_t)fx_face_key_block(k1) * FX_BF_COUNT +
            ((size_t)d * FX_NSTAGES + slot) * FX_NFACES, fx_face_key_idx(k1));
        v[d] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y + b.y));
    }
    const int b = FX_CELL_BLOCK(op.dst);
    const int c = FX_CELL_IDX(op.dst);
    if (fx_nonfinite(v[0].x) || fx_nonfinite(v[1].x) || fx_nonfinite(v[2].x)) {
        fx_fail(D.err, FX_ERR_B_NONFINITE, b, c);
    }
    if (fx_nonfinite(v[0].y) || fx_nonfinite(v[1].y) || fx_nonfinite(v[2].y)) {
        fx_fail(D.err, FX_ERR_B_NONFINITE, b, c + 1);
    }
    double *W = D.W + (size_t)b * FX_W_COUNT(9) + (size_t)slot * FX_NCELLS;
    fx_store2(W + (size_t)FX_B1 * kPlane, c, v[0]);
    fx_store2(W + (size_t)FX_B2 * kPlane, c, v[1]);
    fx_store2(W + (size_t)FX_B3 * kPlane, c, v[2]);
}

/* face-prolongation groups of one wave (a separate kernel: the group
 * arithmetic would otherwise raise the register count, and so lower the
 * occupancy, of the copy-dominated wave kernel) */
__global__ void __launch_bounds__(128) k_ghost_groups(FxDev D, const FxPop *__restrict__ pops, int np, int slot)
{
    if (D.ctl->skip) {
        return;
    }
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 2;
    fx_ghost_prolong_group(D, pops[min(g, np - 1)], slot, g < np);
}

/* face pairs per thread of the wave kernel */
constexpr int FX_GW_FACE_PAIRS = 4;

/* CTAs of each list of a wave */
struct FxWaveGrid {
    int cp, cg, fp, fg, b;
};

/* One conflict-free wave of the ghost fill: the lists of FxWave one after the
 * other, a range of CTAs each.  Bound by DRAM and latency.
 * 512 blocks 149 us (148 with one 16-byte entry per element),
 * 105 blocks 24.7 (30.9), the 470-block blast's fill 288 (314; its groups run
 * beside).  Pairs and single copies in lists of their own, each a pass over the
 * mesh, measured 190 us: they share sectors. */
template <bool BJ>
__global__ void __launch_bounds__(256, BJ ? 4 : 6) k_ghost_wave(FxDev D, FxWave w, FxWaveGrid g, int slot)
{
    if (D.ctl->skip) {
        return;
    }
    int blk = blockIdx.x;
    if (blk < g.cp) {
        const int t = blk * 256 + threadIdx.x;
        if (t < w.ncp) fx_ghost_cell_copy(D, w.cp[t], slot);
        return;
    }
    blk -= g.cp;
    if (blk < g.fp) {
        /* pairs t0 + 256 u: every load first, then the stores */
        constexpr int UP = FX_GW_FACE_PAIRS;
        const int t0 = blk * 256 * UP + threadIdx.x;
        double2 v[UP];
        FxPair op[UP];
#pragma unroll
        for (int u = 0; u < UP; ++u) {
            if (t0 + 256 * u < w.nfp) op[u] = w.fp[t0 + 256 * u];
        }
#pragma unroll
        for (int u = 0; u < UP; ++u) {
            if (t0 + 256 * u < w.nfp) {
                int f;
                const double *p = fx_pair_faces(D, op[u].src, slot, f);
                if (op[u].dst < 0) v[u].x = p[f];
                else v[u] = fx_load2(p, f);
            }
        }
#pragma unroll
        for (int u = 0; u < UP; ++u) {
            if (t0 + 256 * u < w.nfp) {
                int f;
                double *p = fx_pair_faces(D, op[u].dst, slot, f);
                if (op[u].dst < 0) p[f] = v[u].x;
                else fx_store2(p, f, v[u]);
            }
        }
        return;
    }
    blk -= g.fp;
    if (blk < g.b) {
        const int t = blk * 256 + threadIdx.x;
        if (t < w.nb) {
            const FxBop op = w.b[t];
            if (op.pad == 2) fx_ghost_b_pair(D, op, slot);
            else fx_ghost_b_op(D, op, slot);
        }
        return;
    }
    blk -= g.b;
    if (blk < g.cg) {
        const int t = blk * 256 + threadIdx.x;
        if (t < w.ncg) fx_ghost_cell_op<BJ>(D, w.cg[t], slot);
        return;
    }
    blk -= g.cg;
    /* operations t0 + 256 u, u < UF: every load first, then the stores */
    constexpr int UF = FX_GW_FACE_OPS;
    const int t0 = blk * 256 * UF + threadIdx.x;
    double v[UF];
    double *dst[UF];
#pragma unroll
    for (int u = 0; u < UF; ++u) {
        const int t = t0 + 256 * u;
        dst[u] = t < w.nfg ? fx_ghost_face_value(D, w.fg[t], slot, v[u]) : nullptr;
    }
#pragma unroll
    for (int u = 0; u < UF; ++u) {
        if (dst[u]) *dst[u] = v[u];
    }
}

/* component v of block b's flux entry given as direction * nv * cells + AoSoA
 * index of component 0: a face of the block itself (corrections and
 * exchanges reach no other) */
__device__ __forceinline__ double *fx_flux_entry(const FxDev &D, int b, int entry, int v)
{
    const int nv = D.nv;
    const int dir = entry / (nv * FX_NCELLS);
    const int r = entry - dir * nv * FX_NCELLS;
    const int u = r / (FX_AOSOA_W * nv);
    const int row = u / FX_AOSOA_KT;
    const int k = (u - row * FX_AOSOA_KT) * FX_AOSOA_W + r % FX_AOSOA_W - FX_NG;
    const int i = row / FX_PBS - FX_NG;
    const int j = row % FX_PBS - FX_NG;
    if (v >= 6) return D.cx + (size_t)b * FX_CX_COUNT + fx_cx_field(dir, v, i, j, k);
    return D.cf + (size_t)b * FX_CF_COUNT + fx_cf_idx(dir, i, j, k) + v * fx_cf_plane(dir);
}

/* exchanges of a sharded mesh: one thread per listed element */
__device__ __forceinline__ double *fx_xelem(const FxDev &D, const FxXent &x, int slot, int q)
{
    switch (x.kind) {
    case 0:
        return D.W + (size_t)x.block * FX_W_COUNT(D.nv) + (size_t)slot * FX_NCELLS + (size_t)q * kPlane + x.idx;
    case 1: {
        const int dir = x.idx / FX_NFACES;
        return D.Bf + (size_t)x.block * FX_BF_COUNT + ((size_t)dir * FX_NSTAGES + slot) * FX_NFACES +
            (x.idx - dir * FX_NFACES);
    }
    case 2:
        return fx_flux_entry(D, x.block, x.idx, q);
    default:
        return D.emf + (size_t)x.block * FX_EMF_COUNT + x.idx;
    }
}

__device__ __forceinline__ int fx_xwidth(int kind) { return kind == 0 || kind == 2 ? 6 : 1; }

__global__ void k_xpack(FxDev D, const FxXent *__restrict__ ents, int n, double *__restrict__ buf, int slot)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const FxXent x = ents[t];
    for (int q = 0; q < fx_xwidth(x.kind); ++q) buf[x.off + q] = *fx_xelem(D, x, slot, q);
}

__global__ void k_xunpack(FxDev D, const FxXent *__restrict__ ents, int n, const double *__restrict__ buf, int slot)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const FxXent x = ents[t];
    for (int q = 0; q < fx_xwidth(x.kind); ++q) *fx_xelem(D, x, slot, q) = buf[x.off + q];
}

/* coarse/fine corrections */
__global__ void k_flux_correct(FxDev D, const FxCorr *__restrict__ recs, int n, int ncomp)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * ncomp || D.ctl->skip) {
        return;
    }
    const int r = t / ncomp;
    const int v = t - r * ncomp;
    const FxCorr rec = recs[r];
    /* sum order of src/prj_riemann.c:1756-1761 */
    double f[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        f[q] = *fx_flux_entry(D, rec.src_block, rec.src[q], v);
    }
    *fx_flux_entry(D, rec.dst_block, rec.dst, v) = 0.25 * (f[0] + f[1] + f[2] + f[3]);
}

__global__ void k_emf_correct(FxDev D, const FxCorr *__restrict__ recs, int n)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n || D.ctl->skip) {
        return;
    }
    const FxCorr rec = recs[t];
    const double *s = D.emf + (size_t)rec.src_block * FX_EMF_COUNT;
    /* value = 0; value += e0; value += e1; value *= 0.5 (src/prj_mhd.c:904-910):
     * the leading 0.0 + makes a -0.0 pair sum to +0.0 */
    double value = 0.0;
    value += s[rec.src[0]];
    value += s[rec.src[1]];
    value *= 0.5;
    D.emf[(size_t)rec.dst_block * FX_EMF_COUNT + rec.dst] = value;
}

} /* namespace */


/* ------------------------------------------------------------------------ */
/* eSSPRK stored states (prj_timeint_eSSPRK_save_state / _blend_with_saved,  */
/* src/prj_timeint.c:2311-2444)                                              */
/* ------------------------------------------------------------------------ */

__device__ __forceinline__ double *fx_saved_w(const FxDev &D, int b, int which)
{
    return which == 1 ? D.W + (size_t)b * FX_W_COUNT(D.nv) + FX_NCELLS
                      : D.W2 + (size_t)b * D.nv * FX_NCELLS;
}

/* saved face array of direction d: stride of its faces is FX_NFACES */
__device__ __forceinline__ double *fx_saved_bf(const FxDev &D, int b, int d, int which)
{
    return which == 1 ? D.Bf + (size_t)b * FX_BF_COUNT + ((size_t)d * FX_NSTAGES + 1) * FX_NFACES
                      : D.Bf2 + ((size_t)b * 3 + d) * FX_NFACES;
}

/* W of the active cells (all variables) and every face of slot 0 */
__global__ void k_essprk_save(FxDev D, const int *__restrict__ blist, int which)
{
    if (D.ctl->skip) {
        return;
    }
    const int b = blist[blockIdx.y];
    const int nv = D.nv;
    const int ncell = FX_BS * FX_BS * FX_BS;
    const int nface = D.Bf ? 3 * FX_NFACES : 0;
    const double *W0 = D.W + (size_t)b * FX_W_COUNT(nv);
    double *Ws = fx_saved_w(D, b, which);
    const size_t wstride = which == 1 ? (size_t)FX_NSTAGES * FX_NCELLS : (size_t)FX_NCELLS;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nv * ncell + nface; t += gridDim.x * blockDim.x) {
        if (t < nv * ncell) {
            const int v = t / ncell;
            const int r = t - v * ncell;
            const int c = fx_lidx(r >> 8, (r >> 4) & 15, r & 15);
            Ws[(size_t)v * wstride + c] = W0[(size_t)v * kPlane + c];
        } else {
            const int q = t - nv * ncell;
            const int d = q / FX_NFACES;
            const int f = q - d * FX_NFACES;
            fx_saved_bf(D, b, d, which)[f] = D.Bf[(size_t)b * FX_BF_COUNT + (size_t)d * FX_NSTAGES * FX_NFACES + f];
        }
    }
}

/* prj_timeint_eSSPRK_blend_bf: active faces of slot 0 <- w saved + (1 - w) slot 0 */
__global__ void __launch_bounds__(128) k_essprk_blend_faces(FxDev D, const int *__restrict__ blist, int which,
    double w)
{
    if (D.ctl->skip) {
        return;
    }
    const int b = blist[blockIdx.y];
    constexpr int NF = (FX_BS + 1) * FX_BS * FX_BS;
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * NF) {
        return;
    }
    const int dir = t / NF;
    t -= dir * NF;
    const int x2 = dir == 2 ? FX_BS + 1 : FX_BS;
    const int x1 = dir == 1 ? FX_BS + 1 : FX_BS;
    const int k = t % x2;
    t /= x2;
    const int j = t % x1;
    const int i = t / x1;
    const int f = fx_face_idx(dir, i, j, k);
    const double cw = 1.0 - w;
    double *bf0 = D.Bf + (size_t)b * FX_BF_COUNT + (size_t)dir * FX_NSTAGES * FX_NFACES;
    bf0[f] = w * fx_saved_bf(D, b, dir, which)[f] + cw * bf0[f];
}

/* prj_timeint_eSSPRK_final_cell: conserved blend, field from the blended
 * faces, cons2prim into slot 0 */
template <bool MHD>
__global__ void __launch_bounds__(128) k_essprk_blend_cells(FxDev D, const int *__restrict__ blist, int which,
    double w)
{
    if (D.ctl->skip) {
        return;
    }
    const int b = blist[blockIdx.y];
    constexpr int nv = MHD ? 9 : 6;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= FX_BS * FX_BS * FX_BS) {
        return;
    }
    const int i = t >> 8, j = (t >> 4) & 15, k = t & 15;
    const int c = fx_lidx(i, j, k);
    double *W0 = D.W + (size_t)b * FX_W_COUNT(nv);
    const double *Ws = fx_saved_w(D, b, which);
    const size_t wstride = which == 1 ? (size_t)FX_NSTAGES * FX_NCELLS : (size_t)FX_NCELLS;
    const double cw = 1.0 - w;
    double x[9], u[9], us[9];
#pragma unroll
    for (int v = 0; v < nv; ++v) x[v] = W0[(size_t)v * kPlane + c];
    fx_prim2cons<MHD>(x, u);
#pragma unroll
    for (int v = 0; v < nv; ++v) x[v] = Ws[(size_t)v * wstride + c];
    fx_prim2cons<MHD>(x, us);
#pragma unroll
    for (int v = 0; v < nv; ++v) u[v] = w * us[v] + cw * u[v];
    if (MHD) {
        /* prj_timeint_mhd_set_cons_b_from_bf (src/prj_timeint.c:498-510) on slot 0 */
        const double *bf = D.Bf + (size_t)b * FX_BF_COUNT;
        const double *b1 = bf;
        const double *b2 = bf + (size_t)1 * FX_NSTAGES * FX_NFACES;
        const double *b3 = bf + (size_t)2 * FX_NSTAGES * FX_NFACES;
        u[FX_B1] = 0.5 * (b1[fx_face_idx(0, i, j, k)] + b1[fx_face_idx(0, i + 1, j, k)]);
        u[FX_B2] = 0.5 * (b2[fx_face_idx(1, i, j, k)] + b2[fx_face_idx(1, i, j + 1, k)]);
        u[FX_B3] = 0.5 * (b3[fx_face_idx(2, i, j, k)] + b3[fx_face_idx(2, i, j, k + 1)]);
        if (!isfinite(u[FX_B1]) || !isfinite(u[FX_B2]) || !isfinite(u[FX_B3])) {
            fx_fail(D.err, FX_ERR_B_NONFINITE, b, c);
        }
    }
    fx_cons2prim<MHD>(u, x);
#pragma unroll
    for (int v = 0; v < nv; ++v) W0[(size_t)v * kPlane + c] = x[v];
}

/* ------------------------------------------------------------------------ */
/* launchers                                                                 */
/* ------------------------------------------------------------------------ */
static inline unsigned fx_blocks(int n, int tpb) { return (unsigned)((n + tpb - 1) / tpb); }

/* launch shapes of the face kernel: {threads per CTA, min CTAs per SM} */
static const int kFluxShapes[FX_FLUX_VARIANTS][2] = {{64, 9}, {64, 8}, {32, 18}, {128, 5}, {64, 12}, {256, 3}};

using FxFluxKernel = void (*)(FxDev, const int *, int, int);
struct FxFluxLaunch {
    FxFluxKernel fn;
    int tpb;
};

/* the autotuner's launch shapes (threads per CTA, minimum CTAs per SM).
 * Microseconds per launch, MC / WENO-Z3 / hydro MC (512, 216, 216 blocks):
 * 64 x 9  505 / 607 / 101    32 x 18  503 / 612 / 101    64 x 8  535 / 622 / 108
 * 128 x 5 550 / 592 / 103    64 x 12  534 / 557 / 93     256 x 3 563 / 536 / 97
 * 18 warps per SM at 96 registers suit MC; WENO-Z3 with 48 divisions per face
 * in its reconstruction wants the 24 warps of 80 registers; small CTAs leave
 * no half-empty SM behind a slow warp. */
template <bool MHD, bool FULL, bool RING, int RECON>
static FxFluxLaunch flux_shape(int variant)
{
    if constexpr (FULL) {
        /* the plain form's launches hold one block, 258 CTAs of 64: two per
         * SM whatever the shape allows, so the one that does not spill */
        return {k_flux<MHD, true, true, 64, 8, RECON>, 64};
    } else {
        switch (variant) {
        case 1: return {k_flux<MHD, false, RING, 64, 8, RECON>, 64};
        case 2: return {k_flux<MHD, false, RING, 32, 18, RECON>, 32};
        case 3: return {k_flux<MHD, false, RING, 128, 5, RECON>, 128};
        case 4: return {k_flux<MHD, false, RING, 64, 12, RECON>, 64};
        case 5: return {k_flux<MHD, false, RING, 256, 3, RECON>, 256};
        default: return {k_flux<MHD, false, RING, 64, 9, RECON>, 64};
        }
    }
}

/* Every reconstruction is compiled in every launch shape.  WENO-Z7 reads
 * three cells beyond each face's neighbours and exists in the
 * four-ghost-layer build only (the context rejects it elsewhere); its
 * register demand (about 180 per thread unbounded) makes the shape matter. */
template <bool MHD, bool FULL, bool RING>
static FxFluxLaunch flux_kernel(const FxDev &D)
{
    if (D.recon == FX_RECON_WENO3) return flux_shape<MHD, FULL, RING, FX_RECON_WENO3>(D.flux_variant);
#if FX_NG >= 4
    if (D.recon == FX_RECON_WENO7) return flux_shape<MHD, FULL, RING, FX_RECON_WENO7>(D.flux_variant);
#endif
    return flux_shape<MHD, FULL, RING, FX_RECON_MC>(D.flux_variant);
}

static FxFluxLaunch flux_kernel(const FxDev &D, int full, int inner)
{
    if (D.nv != 9) return full ? flux_kernel<false, true, false>(D) : flux_kernel<false, false, false>(D);
    if (full) return flux_kernel<true, true, true>(D);
    return inner ? flux_kernel<true, false, false>(D) : flux_kernel<true, false, true>(D);
}

void *fx_flux_function(const FxDev &D, int inner) { return (void *)flux_kernel(D, 0, inner).fn; }

void fx_launch_flux(const FxDev &D, const int *blist, int nlist, int ndir, int wslot, int bfslot,
    int full, int inner, cudaStream_t s)
{
    if (nlist <= 0) return;
    FxFluxLaunch f = flux_kernel(D, full, inner);
    if (D.br_mode != 0 && full && D.nv == 9 && D.recon == FX_RECON_MC) {
        /* the plain form recording or replaying its decisions */
        f.fn = D.br_mode == 1 ? k_flux<true, true, true, 128, 4, FX_RECON_MC, 1>
                              : k_flux<true, true, true, 128, 4, FX_RECON_MC, 2>;
        f.tpb = 128;
    }
    const int nf = D.nv == 9 ? (FX_BS + 1) * (FX_BS + 2) * (FX_BS + 2) : (FX_BS + 1) * FX_BS * FX_BS;
    f.fn<<<dim3(fx_blocks(nf, f.tpb), ndir, nlist), f.tpb, 0, s>>>(D, blist, wslot, bfslot);
}

void fx_flux_shape(int variant, int *tpb, int *minb)
{
    const int v = variant >= 0 && variant < FX_FLUX_VARIANTS ? variant : 0;
    *tpb = kFluxShapes[v][0];
    *minb = kFluxShapes[v][1];
}

/* ------------------------------------------------------------------------ */
/* Dump payloads (prj_io_write_dump, src/prj_io.c:1994-2330)                */
/* ------------------------------------------------------------------------ */
/* The rows of the dump's Data, Eos and Bf datasets for the listed blocks,
 * packed per list position q at out + q * row: Data [v][cell] (stage slot 0
 * of W, cell = (i * 16 + j) * 16 + k over the active cells), Eos [v][cell]
 * (p, T, gamma from eosvar), then, when faces is set, Bf [d][face] (stage
 * slot 0, all faces). */
__global__ void __launch_bounds__(256) k_dump_pack(FxDev D, const int *__restrict__ blist, int faces,
    double *__restrict__ out)
{
    constexpr int NC = FX_BS * FX_BS * FX_BS;
    const int nv = D.nv;
    const size_t row = (size_t)(nv + 3) * NC + (faces ? (size_t)3 * FX_NFACES : 0);
    const int b = blist[blockIdx.y];
    double *o = out + (size_t)blockIdx.y * row;
    for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < row; t += (size_t)gridDim.x * blockDim.x) {
        if (t < (size_t)(nv + 3) * NC) {
            const int v = (int)(t / NC);
            const int r = (int)(t - (size_t)v * NC);
            const int i = r / (FX_BS * FX_BS), j = (r / FX_BS) % FX_BS, k = r % FX_BS;
            if (v < nv) {
                o[t] = D.W[(size_t)b * FX_W_COUNT(nv) + (size_t)v * FX_NSTAGES * FX_NCELLS + fx_lidx(i, j, k)];
            } else {
                o[t] = D.eos[(size_t)b * FX_EOS_COUNT + fx_bidx(3, v - nv, i, j, k)];
            }
        } else {
            const size_t u = t - (size_t)(nv + 3) * NC;
            const int d = (int)(u / FX_NFACES);
            const int n = (int)(u - (size_t)d * FX_NFACES);
            o[t] = D.Bf[(size_t)b * FX_BF_COUNT + (size_t)d * FX_NSTAGES * FX_NFACES + n];
        }
    }
}

void fx_launch_dump_pack(const FxDev &D, const int *blist, int nlist, int faces, double *out, cudaStream_t s)
{
    if (nlist <= 0) return;
    k_dump_pack<<<dim3(64, nlist), 256, 0, s>>>(D, blist, faces, out);
}

/* ------------------------------------------------------------------------ */
/* Active-region state transfers: the cell-centred field after an upload    */
/* ------------------------------------------------------------------------ */
/* The cell-centred field of the listed blocks' active cells from their
 * faces, stage slot 0: prj_mhd_bf2bc_impl's arithmetic (src/prj_mhd.c:
 * 585-590; the metric factor is 1 outside dynamical GR) */
__global__ void __launch_bounds__(256) k_cell_field_active(FxDev D, const int *__restrict__ blist)
{
    constexpr int NC = FX_BS * FX_BS * FX_BS;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= NC) {
        return;
    }
    const int b = blist[blockIdx.y];
    const int i = t / (FX_BS * FX_BS), j = (t / FX_BS) % FX_BS, k = t % FX_BS;
    const double *bf = D.Bf + (size_t)b * FX_BF_COUNT;
    const double *f1 = bf;
    const double *f2 = bf + (size_t)FX_NSTAGES * FX_NFACES;
    const double *f3 = bf + (size_t)2 * FX_NSTAGES * FX_NFACES;
    const double b1 = 0.5 * (f1[fx_face_idx(0, i, j, k)] + f1[fx_face_idx(0, i + 1, j, k)]);
    const double b2 = 0.5 * (f2[fx_face_idx(1, i, j, k)] + f2[fx_face_idx(1, i, j + 1, k)]);
    const double b3 = 0.5 * (f3[fx_face_idx(2, i, j, k)] + f3[fx_face_idx(2, i, j, k + 1)]);
    if (!isfinite(b1) || !isfinite(b2) || !isfinite(b3)) {
        fx_fail(D.err, FX_ERR_B_NONFINITE, b, fx_lidx(i, j, k));
    }
    double *w = D.W + (size_t)b * FX_W_COUNT(9) + fx_lidx(i, j, k);
    w[(size_t)FX_B1 * FX_NSTAGES * FX_NCELLS] = b1;
    w[(size_t)FX_B2 * FX_NSTAGES * FX_NCELLS] = b2;
    w[(size_t)FX_B3 * FX_NSTAGES * FX_NCELLS] = b3;
}

void fx_launch_cell_field_active(const FxDev &D, const int *blist, int nlist, cudaStream_t s)
{
    if (nlist <= 0) return;
    constexpr int NC = FX_BS * FX_BS * FX_BS;
    k_cell_field_active<<<dim3(fx_blocks(NC, 256), nlist), 256, 0, s>>>(D, blist);
}

/* one block's face arrays in the reference's tiles, for a download */
__global__ void __launch_bounds__(256) k_face_tiles(FxDev D, int b, int dir, int velocities, double *__restrict__ out)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= FX_NCELLS) {
        return;
    }
    if (velocities) {
        for (int v = 0; v < 3; ++v) {
            const int m = (v + 3 - dir) % 3;
            out[fx_bidx_cell(3, v, t)] = m == 0 ? D.vn[(size_t)b * FX_VN_COUNT + dir * FX_NCELLS + t]
                : D.vt[(size_t)b * FX_VT_COUNT + (2 * dir + m - 1) * FX_NCELLS + t];
        }
        return;
    }
    const int i = t / (FX_PBS * FX_PBS) - FX_NG, j = (t / FX_PBS) % FX_PBS - FX_NG, k = t % FX_PBS - FX_NG;
    const bool own = fx_is_face(dir, 0, i, j, k);
    const bool ring = D.nv == 9 && fx_is_face(dir, 1, i, j, k); /* own faces too */
    const double *cf = D.cf + (size_t)b * FX_CF_COUNT;
    const double *cx = D.cx + (size_t)b * FX_CX_COUNT;
    for (int v = 0; v < D.nv; ++v) {
        double f = 0.0;
        if (v >= 6) {
            if (ring) f = cx[fx_cx_field(dir, v, i, j, k)];
        } else if (own) {
            f = cf[fx_cf_idx(dir, i, j, k) + v * fx_cf_plane(dir)];
        } else if (ring) {
            f = cx[fx_cx_idx(dir, i, j, k) + v * fx_cx_plane(dir)];
        }
        out[fx_bidx_cell(D.nv, v, t)] = f;
    }
}

void fx_launch_face_tiles(const FxDev &D, int b, int dir, int velocities, double *out, cudaStream_t s)
{
    k_face_tiles<<<fx_blocks(FX_NCELLS, 256), 256, 0, s>>>(D, b, dir, velocities, out);
}

void fx_launch_emf(const FxDev &D, const int *blist, int nlist, int wslot, int bfslot, cudaStream_t s)
{
    if (nlist <= 0) return;
    if (nlist < 16) {
        const dim3 grid(fx_blocks(3 * FX_BS * (FX_BS + 1) * (FX_BS + 1), 128), nlist);
        k_emf_edges<<<grid, 128, 0, s>>>(D, blist, wslot, bfslot);
        return;
    }
    /* chunks of edge layers: two rounds of the 296 CTAs that fit (two per
     * SM), at least two chunks, since each chunk reads one plane again: 64
     * blocks 20.6 us with 10 chunks, 22.7 with 14 */
    constexpr int fill = 592;
    const int nchunk = nlist * 17 <= fill ? 17 : nlist * 2 >= fill ? 2 : (fill + nlist - 1) / nlist;
    k_emf<<<dim3(nchunk, nlist), kEmfThreads, kEmfSmem, s>>>(D, blist, wslot, bfslot, nchunk);
}

cudaError_t fx_prepare_kernels()
{
    return cudaFuncSetAttribute(k_emf, cudaFuncAttributeMaxDynamicSharedMemorySize, kEmfSmem);
}

void fx_launch_bf_update(const FxDev &D, const int *blist, int nlist, int stage, cudaStream_t s)
{
    if (nlist <= 0) return;
    const int nf = (FX_BS + 1) * FX_BS * FX_BS;
    k_bf_update<<<dim3(fx_blocks(nf, 128), 3, nlist), 128, 0, s>>>(D, blist, stage);
}

template <bool MHD, bool FULL>
static void launch_cell_update(const FxDev &D, const int *blist, int nlist, int stage, int gravity, int next_dt,
    cudaStream_t s)
{
    const dim3 grid(fx_blocks(FX_BS * FX_BS * FX_BS, 128), nlist);
    if (!FULL && stage == 2 && next_dt) k_cell_update<MHD, 2, false, true><<<grid, 128, 0, s>>>(D, blist, gravity);
    else if (stage == 1) k_cell_update<MHD, 1, FULL><<<grid, 128, 0, s>>>(D, blist, gravity);
    else if (stage == 2) k_cell_update<MHD, 2, FULL><<<grid, 128, 0, s>>>(D, blist, gravity);
    else k_cell_update<MHD, 0, FULL><<<grid, 128, 0, s>>>(D, blist, gravity);
}

void fx_launch_cell_update(const FxDev &D, const int *blist, int nlist, int stage,
    int gravity, int full, int next_dt, cudaStream_t s)
{
    if (nlist <= 0) return;
    if (D.nv == 9) {
        if (full) launch_cell_update<true, true>(D, blist, nlist, stage, gravity, next_dt, s);
        else launch_cell_update<true, false>(D, blist, nlist, stage, gravity, next_dt, s);
    } else {
        if (full) launch_cell_update<false, true>(D, blist, nlist, stage, gravity, next_dt, s);
        else launch_cell_update<false, false>(D, blist, nlist, stage, gravity, next_dt, s);
    }
}

void fx_launch_eos_fill(const FxDev &D, const int *blist, int nlist, int wslot, int active_only,
    cudaStream_t s)
{
    if (nlist <= 0) return;
    const int n = active_only ? FX_BS * FX_BS * FX_BS : FX_NCELLS;
    k_eos_fill<<<dim3(fx_blocks(n, 256), nlist), 256, 0, s>>>(D, blist, wslot, active_only);
}

void fx_launch_calc_dt(const FxDev &D, const int *blist, int nlist, int wslot, double cfl,
    cudaStream_t s)
{
    if (nlist <= 0) return;
    k_calc_dt<<<dim3(fx_blocks(FX_BS * FX_BS * FX_BS, 256), nlist), 256, 0, s>>>(D, blist, wslot, cfl);
}

void fx_launch_ghost_wave(const FxDev &D, const FxWave &w, int slot, cudaStream_t s)
{
    const FxWaveGrid g = {(int)fx_blocks(w.ncp, 256), (int)fx_blocks(w.ncg, 256),
        (int)fx_blocks(w.nfp, 256 * FX_GW_FACE_PAIRS), (int)fx_blocks(w.nfg, 256 * FX_GW_FACE_OPS),
        (int)fx_blocks(w.nb, 256)};
    const unsigned grid = (unsigned)(g.cp + g.cg + g.fp + g.fg + g.b);
    if (grid > 0) {
        if (D.use_bj) k_ghost_wave<true><<<grid, 256, 0, s>>>(D, w, g, slot);
        else k_ghost_wave<false><<<grid, 256, 0, s>>>(D, w, g, slot);
    }
}

void fx_launch_xpack(const FxDev &D, const FxXent *ents, int n, double *buf, int slot, cudaStream_t s)
{
    if (n > 0) k_xpack<<<fx_blocks(n, 256), 256, 0, s>>>(D, ents, n, buf, slot);
}

void fx_launch_xunpack(const FxDev &D, const FxXent *ents, int n, const double *buf, int slot, cudaStream_t s)
{
    if (n > 0) k_xunpack<<<fx_blocks(n, 256), 256, 0, s>>>(D, ents, n, buf, slot);
}

void fx_launch_prolong_groups(const FxDev &D, const FxPop *pops, int np, int slot, cudaStream_t s)
{
    if (np > 0) {
        k_ghost_groups<<<fx_blocks(4 * np, 128), 128, 0, s>>>(D, pops, np, slot);
    }
}

void fx_launch_flux_correct(const FxDev &D, const FxCorr *recs, int n, int ncomp, cudaStream_t s)
{
    if (n <= 0) return;
    k_flux_correct<<<fx_blocks(n * ncomp, 256), 256, 0, s>>>(D, recs, n, ncomp);
}

void fx_launch_emf_correct(const FxDev &D, const FxCorr *recs, int n, cudaStream_t s)
{
    if (n <= 0) return;
    k_emf_correct<<<fx_blocks(n, 256), 256, 0, s>>>(D, recs, n);
}

void fx_launch_reset_reductions(const FxDev &D, int which, cudaStream_t s)
{
    k_reset_reductions<<<1, 1, 0, s>>>(D, which);
}

void fx_launch_step_begin(const FxDev &D, cudaStream_t s)
{
    k_step_begin<<<1, 1, 0, s>>>(D);
}

void fx_launch_step_end(const FxDev &D, cudaStream_t s)
{
    k_step_end<<<1, 1, 0, s>>>(D);
}

namespace {
__global__ void k_set_dt(FxDev D, double dt)
{
    D.ctl->dt = dt;
    D.ctl->dt_stage = dt;
    D.ctl->skip = 0;
}

__global__ void k_stage_dt(FxDev D, double divisor)
{
    D.ctl->dt_stage = D.ctl->dt / divisor;
}

__global__ void k_set_ctl(FxDev D, FxCtl v)
{
    *D.ctl = v;
}
}

void fx_launch_set_dt(const FxDev &D, double dt, cudaStream_t s)
{
    k_set_dt<<<1, 1, 0, s>>>(D, dt);
}

void fx_launch_stage_dt(const FxDev &D, double divisor, cudaStream_t s)
{
    k_stage_dt<<<1, 1, 0, s>>>(D, divisor);
}

void fx_launch_essprk_save(const FxDev &D, const int *blist, int nlist, int which, cudaStream_t s)
{
    if (nlist <= 0) return;
    k_essprk_save<<<dim3(32, nlist), 256, 0, s>>>(D, blist, which);
}

void fx_launch_essprk_blend(const FxDev &D, const int *blist, int nlist, int which, double w, cudaStream_t s)
{
    if (nlist <= 0) return;
    if (D.nv == 9) {
        const int nf = 3 * (FX_BS + 1) * FX_BS * FX_BS;
        k_essprk_blend_faces<<<dim3(fx_blocks(nf, 128), nlist), 128, 0, s>>>(D, blist, which, w);
        k_essprk_blend_cells<true><<<dim3(fx_blocks(FX_BS * FX_BS * FX_BS, 128), nlist), 128, 0, s>>>(
            D, blist, which, w);
    } else {
        k_essprk_blend_cells<false><<<dim3(fx_blocks(FX_BS * FX_BS * FX_BS, 128), nlist), 128, 0, s>>>(
            D, blist, which, w);
    }
}

void fx_launch_set_ctl(const FxDev &D, FxCtl value, cudaStream_t s)
{
    k_set_ctl<<<1, 1, 0, s>>>(D, value);
}
