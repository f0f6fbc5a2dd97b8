/*
 * Per-block memory layout of the device mirror.
 *
 * The device keeps every block array in exactly the reference's per-block
 * layout so that offsets agree between a host prj_block and its device copy:
 *   - block geometry: BLOCK_SIZE=16 active cells, NGHOST=2, so 20 cells per
 *     axis with ghosts (reference src/prj_defs.h:383-388);
 *   - LIDX: untiled cell index, k fastest (src/prj_defs.h:392-393);
 *   - FACE_IDX / EDGE_IDX: staggered face and edge indices, one extra point
 *     along the staggered axis (src/prj_defs.h:394-405);
 *   - BIDX: AoSoA cell buffers [i][j][k/4][var][k%4] with lane width 4
 *     (src/prj_defs.h:419-434), used by flux, v_riemann, eosvar, rhs;
 *   - WIDX: primitives stage-major per variable, v*NSTAGES*NCELLS + cell
 *     (src/prj_defs.h:451-453).
 * These index formulas are the interface the drop-in must honour, so they
 * are restated here with the same meaning.  Blocks are stacked: block b's
 * array starts at base + b * per_block_count.
 */
#ifndef FX_LAYOUT_H
#define FX_LAYOUT_H

#ifdef __CUDACC__
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD inline
#endif

#define FX_BS 16
#ifndef FX_NG
#define FX_NG 2                              /* 4 for the WENO-Z7 build (PRJ_NGHOST) */
#endif
#define FX_PBS (FX_BS + 2 * FX_NG)          /* 20 */
#define FX_NCELLS (FX_PBS * FX_PBS * FX_PBS) /* 8000 */
#define FX_NFACES ((FX_PBS + 1) * FX_PBS * FX_PBS) /* 8400 */
#define FX_NEDGES ((FX_PBS + 1) * (FX_PBS + 1) * FX_PBS) /* 8820 */
#define FX_NSTAGES 2
#define FX_AOSOA_W 4
#define FX_AOSOA_KT (FX_PBS / FX_AOSOA_W) /* 5 */
#define FX_NSLOTS 56
#define FX_MAXVAR 9

/* primitive / conserved variable slots (src/prj_defs.h:466-494) */
#define FX_RHO 0
#define FX_V1 1
#define FX_V2 2
#define FX_V3 3
#define FX_EINT 4
#define FX_ETOT 4
#define FX_YE 5
#define FX_B1 6
#define FX_B2 7
#define FX_B3 8

/* eosvar components */
#define FX_EOS_P 0
#define FX_EOS_T 1
#define FX_EOS_G 2

/* ideal-gas temperature scale of the reference's ideal EOS provider */
#define FX_IDEAL_ENERGY_SCALE 0.95655684e18

FX_HD int fx_lidx(int i, int j, int k)
{
    return ((i + FX_NG) * FX_PBS + (j + FX_NG)) * FX_PBS + (k + FX_NG);
}

FX_HD int fx_face_idx(int dir, int i, int j, int k)
{
    return dir == 0 ? ((i + FX_NG) * FX_PBS * FX_PBS + (j + FX_NG) * FX_PBS + (k + FX_NG))
         : dir == 1 ? ((i + FX_NG) * (FX_PBS + 1) * FX_PBS + (j + FX_NG) * FX_PBS + (k + FX_NG))
                    : ((i + FX_NG) * FX_PBS * (FX_PBS + 1) + (j + FX_NG) * (FX_PBS + 1) + (k + FX_NG));
}

FX_HD int fx_edge_idx(int dir, int i, int j, int k)
{
    return dir == 0 ? ((i + FX_NG) * (FX_PBS + 1) * (FX_PBS + 1) + (j + FX_NG) * (FX_PBS + 1) + (k + FX_NG))
         : dir == 1 ? ((i + FX_NG) * FX_PBS * (FX_PBS + 1) + (j + FX_NG) * (FX_PBS + 1) + (k + FX_NG))
                    : ((i + FX_NG) * (FX_PBS + 1) * FX_PBS + (j + FX_NG) * FX_PBS + (k + FX_NG));
}

/* AoSoA index of component v of an nc-component cell buffer */
FX_HD int fx_bidx(int nc, int v, int i, int j, int k)
{
    const int kk = k + FX_NG;
    return ((((i + FX_NG) * FX_PBS + (j + FX_NG)) * FX_AOSOA_KT + kk / FX_AOSOA_W) * nc + v) *
        FX_AOSOA_W + kk % FX_AOSOA_W;
}

/* same AoSoA index from an untiled cell index */
FX_HD int fx_bidx_cell(int nc, int v, int cell)
{
    const int row = cell / FX_PBS;
    const int kk = cell - row * FX_PBS;
    return ((row * FX_AOSOA_KT + kk / FX_AOSOA_W) * nc + v) * FX_AOSOA_W + kk % FX_AOSOA_W;
}

/* Face arrays.  Both forms keep theirs in the same four arrays, laid out for
 * the kernels that read them; a download puts them into the reference's
 * VIDX / VRIDX tiles.
 *
 * cf: fluxes of variables 0-5, [dir][variable][i][j][k]: the faces of
 * the block itself only, in rows of 16 (20 along the sweep direction 2, 17 of
 * them used), so rows start on 32-byte sectors and a variable's plane is
 * read end to end. */
#define FX_CF_PLANE ((FX_BS + 1) * FX_BS * FX_BS)       /* directions 0 and 1 */
#define FX_CF_ROW2 (FX_BS + 4)
#define FX_CF_PLANE2 (FX_BS * FX_BS * FX_CF_ROW2)
#define FX_CF_COUNT (12 * FX_CF_PLANE + 6 * FX_CF_PLANE2)

FX_HD int fx_cf_plane(int dir) { return dir == 2 ? FX_CF_PLANE2 : FX_CF_PLANE; }

/* variable 0 of a face; variable v sits v planes further */
FX_HD int fx_cf_idx(int dir, int i, int j, int k)
{
    return dir * 6 * FX_CF_PLANE + (dir == 0 ? (i * FX_BS + j) * FX_BS + k
                                  : dir == 1 ? (i * (FX_BS + 1) + j) * FX_BS + k
                                             : (i * FX_BS + j) * FX_CF_ROW2 + k);
}

/* cx (MHD): the fluxes no later phase reads.  First variables 0-5 on the
 * transverse ghost layer of faces that the EMFs need, [dir][variable][s][r]
 * ([r][s] along direction 2, rows of 20), s along the sweep and r around the
 * block: the rows at -1 and 16 of the first transverse axis, then the
 * columns at -1 and 16 of the second.  Then the field components, which the
 * plain form alone stores, [dir][component][i][j][k] with the ghost layer. */
#define FX_CX_RING (4 * (FX_BS + 1))
#define FX_CX_PLANE (FX_CX_RING * (FX_BS + 1))          /* directions 0 and 1 */
#define FX_CX_PLANE2 (FX_CX_RING * FX_CF_ROW2)
#define FX_CX_FIELD (12 * FX_CX_PLANE + 6 * FX_CX_PLANE2)
#define FX_CX_BOX ((FX_BS + 1) * (FX_BS + 2) * (FX_BS + 2))
#define FX_CX_COUNT (FX_CX_FIELD + 9 * FX_CX_BOX)

FX_HD int fx_cx_plane(int dir) { return dir == 2 ? FX_CX_PLANE2 : FX_CX_PLANE; }

/* variable 0 of a face of the ghost layer */
FX_HD int fx_cx_idx(int dir, int i, int j, int k)
{
    const int s = dir == 0 ? i : dir == 1 ? j : k;
    const int a = dir == 0 ? j : i, b = dir == 2 ? j : k;
    const int r = a < 0 ? b + 1 : a == FX_BS ? FX_BS + 3 + b : (b < 0 ? 2 : 3) * FX_BS + 4 + a;
    return dir * 6 * FX_CX_PLANE + (dir == 2 ? r * FX_CF_ROW2 + s : s * FX_CX_RING + r);
}

/* field component v (6-8) of a face, ghost layer or not */
FX_HD int fx_cx_field(int dir, int v, int i, int j, int k)
{
    const int ej = dir == 1 ? FX_BS + 1 : FX_BS + 2, ek = dir == 2 ? FX_BS + 1 : FX_BS + 2;
    return FX_CX_FIELD + (3 * dir + v - 6) * FX_CX_BOX +
        ((i + (dir != 0)) * ej + j + (dir != 1)) * ek + k + (dir != 2);
}

/* whether (i, j, k) is a face of direction dir of the block itself (ring 0),
 * or one of these or of the transverse ghost layer (ring 1) */
FX_HD bool fx_is_face(int dir, int ring, int i, int j, int k)
{
    const int n = FX_BS + 2 * ring;
    return (dir == 0 ? (unsigned)i < FX_BS + 1u : (unsigned)(i + ring) < (unsigned)n) &&
        (dir == 1 ? (unsigned)j < FX_BS + 1u : (unsigned)(j + ring) < (unsigned)n) &&
        (dir == 2 ? (unsigned)k < FX_BS + 1u : (unsigned)(k + ring) < (unsigned)n);
}

/* per-block element counts of the stacked device arrays: vn the face
 * velocities along the sweep, [dir][cell], vt the transverse ones (plain
 * form), [dir][2][cell] with component (dir + 1 + m) % 3 at m */
#define FX_W_COUNT(nv) ((nv) * FX_NSTAGES * FX_NCELLS)
#define FX_BF_COUNT (3 * FX_NSTAGES * FX_NFACES)
#define FX_VN_COUNT (3 * FX_NCELLS)
#define FX_VT_COUNT (6 * FX_NCELLS)
#define FX_BV_COUNT (3 * FX_NCELLS)
#define FX_EMF_COUNT (3 * FX_NEDGES)
#define FX_EOS_COUNT (3 * FX_NCELLS)
#define FX_RHS_COUNT(nv) ((nv) * FX_NCELLS)
#define FX_GRAV_COUNT (3 * FX_NCELLS)

#endif
