/*
 * Host check of the face kernel's solver (fornaxamr_b200/csrc/fx_physics.cuh)
 * against the plain-C restatement (oracle/fx_oracle.c), double for double:
 * the halved MC slope, WENO face values of one side against those of both,
 * HLLD with the cheap checks and with the checks themselves, and with the
 * internal energy and composition of the near side alone, HLLC.  States are seeded: ordinary ones, every fan region, and
 * broken ones (negative, zero, subnormal, infinite and NaN entries, nearly
 * cancelled waves); a face that the solver's checks reject must never pass
 * the cheap ones.
 */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include "fx_physics.cuh"

extern "C" {
double fxo_mc_slope(double qm, double q0, double qp);
double fxo_weno3_face(double qm, double q0, double qp, double target);
int fxo_hlld(const double *WL, const double *WR, double pL, double pR, double gL, double gR, double bn, double *out);
void fxo_hllc(const double *WL, const double *WR, double pL, double pR, double gL, double gR, double du, double dv,
    double dw, double *out);
}

static uint64_t st = 88172645463325252ULL;
static uint64_t rnd()
{
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return st;
}
static double uni() { return (double)(rnd() >> 11) * (1.0 / 9007199254740992.0); }
static double sym() { return 2.0 * uni() - 1.0; }

static bool same(double a, double b)
{
    if (a != a && b != b) return true;
    return memcmp(&a, &b, sizeof a) == 0;
}

static long bad = 0;
static void expect(bool ok, const char *what, long n)
{
    if (!ok && ++bad < 20) printf("%s differs in case %ld\n", what, n);
}

/* values where comparisons, scaling by two and products can go wrong; up to
 * 2^1022, so that no difference of two is infinite */
static double edge()
{
    static const double v[] = {0.0, -0.0, 1.0, -1.0, 1.0 + 0x1p-52, 1.0 - 0x1p-53, 0x1p-1074, 0x1.8p-1073, 0x1p-1022,
        0x1p-538, 0x1.fp-537, 0x1p-500, 1e-170, 1e-300, 1e300, 0x1p1021, 3.0, 1.0 / 3.0};
    const double x = v[rnd() % (sizeof v / sizeof v[0])];
    return rnd() & 1 ? -x : x;
}

static void state(double *w, double &p, int kind)
{
    const double m = kind == 1 ? 3.0 : kind == 2 ? 0.05 : 0.6; /* supersonic, near rest, ordinary */
    w[0] = 0.1 + uni();
    for (int v = 1; v < 4; ++v) w[v] = m * sym();
    w[4] = 0.2 + uni();
    w[5] = uni();
    for (int v = 6; v < 9; ++v) w[v] = (kind == 3 ? 1e-6 : 0.7) * sym();
    p = (2.0 / 3.0) * w[0] * w[4] * (1.0 + 0.1 * sym());
}

static double broken()
{
    static const double v[] = {0.0, -0.0, -1.0, -1e-3, 0x1p-1074, -0x1p-1040, 0x1p-1030, INFINITY, -INFINITY, NAN, -NAN, 1e300,
        -1e300, 1e-300, 1e160, 1e-160};
    return v[rnd() % (sizeof v / sizeof v[0])];
}

/* the value of one side, read from memory with a stride as the face kernel
 * does, against both sides' from the stencil's values */
template <int RECON>
static void one_side(long i)
{
    constexpr int NS = FxStencil<RECON>::NS;
    static const int strides[] = {1, 20, 400, 24, 576};
    static double mem[7 * 576 + 1];
    const int s = strides[rnd() % 5];
    double q[NS], wl, wr;
    const double base = sym() * exp(10.0 * sym());
    for (int n = 0; n < NS; ++n) {
        q[n] = i % 3 == 0 ? base : i % 3 == 1 ? base * (1.0 + 0.1 * sym()) : edge() * 0x1p-200;
        if (i % 5 == 0 && n > 0 && rnd() % 2) q[n] = q[n - 1];
    }
    for (double &x : mem) x = NAN; /* nothing beside the stencil is read */
    for (int n = 0; n < NS; ++n) mem[n * s] = q[n];
    fx_recon_pair<RECON>(q, wl, wr);
    expect(same(fx_recon_one<RECON>(mem, s, true), wl) && same(fx_recon_one<RECON>(mem, s, false), wr),
        RECON == FX_RECON_WENO7 ? "WENO-Z7 side" : "WENO-Z3 side", i);
    if (RECON == FX_RECON_WENO3) {
        expect(same(wl, fxo_weno3_face(q[0], q[1], q[2], 0.5)) && same(wr, fxo_weno3_face(q[1], q[2], q[3], -0.5)),
            "WENO-Z3 value", i);
    }
}

int main()
{
    const long n = 400000;
    for (long i = 0; i < n; ++i) {
        double q[3];
        for (double &x : q) x = i % 2 ? edge() : sym() * exp(20.0 * sym());
        if (i % 7 == 0) q[2] = q[1] + (q[1] - q[0]) * (i % 3 ? 1.0 : 3.0);
        const double s = 0.5 * fxo_mc_slope(q[0], q[1], q[2]);
        const double h = fx_mc_half(q[1] - q[0], q[2] - q[1]);
        expect(same(q[1] + s, q[1] + h) && same(q[1] - s, q[1] - h), "MC slope", i);
        /* the scaling argument: magnitudes at the subnormal end of a product */
        const double a = ldexp(1.0 + uni(), -(int)(rnd() % 1070)), b = ldexp(1.0 + uni(), -(int)(rnd() % 1070));
        expect(same(0.5 * fxo_mc_slope(-a, 0.0, b), fx_mc_half(a, b)), "MC slope (small)", i);
        expect(same(0.5 * fxo_mc_slope(a, 0.0, -b), fx_mc_half(-a, -b)), "MC slope (small, negative)", i);
        if (i % 4 == 0) {
            one_side<FX_RECON_WENO3>(i / 4);
            one_side<FX_RECON_WENO7>(i / 4);
        }
    }
    long one = 0, rejected = 0, suspected = 0, sound = 0, doubtful = 0;
    for (long i = 0; i < n; ++i) {
        double WL[9], WR[9], pL, pR, bn = (i % 5 == 4 ? 1e-7 : 0.7) * sym(), g = 5.0 / 3.0;
        state(WL, pL, (int)(rnd() % 4));
        if (i % 4 == 0) {
            memcpy(WR, WL, sizeof WR);
            pR = pL;
            for (double &x : WR) x *= 1.0 + 1e-3 * sym();
        } else {
            state(WR, pR, (int)(rnd() % 4));
        }
        const bool brk = i % 10 == 9;
        if (brk) {
            double *at[] = {WL, WR, &pL, &pR, &bn, WL + 1, WR + 1, WL + 4, WR + 7, WL + 8};
            const int k = (int)(rnd() % 10);
            *at[k] = broken();
            if (rnd() % 4 == 0) *at[rnd() % 10] = broken();
        }
        WL[6] = WR[6] = bn;
        FxBrFree br;
        FxFaceOut a, b;
        memset(&a, 0, sizeof a);
        memset(&b, 0, sizeof b);
        FxSuspect sus;
        FxErrLocal le;
        fx_riemann_hlld_folded_br(WL, WR, pL, pR, g, g, bn, a, &sus, 1, 2, br);
        fx_riemann_hlld_folded_br(WL, WR, pL, pR, g, g, bn, b, &le, 1, 2, br);
        expect(memcmp(&a, &b, sizeof a) == 0 || brk, "HLLD policies", i);
        for (int v = 0; v < 9; ++v) expect(same(a.F[v], b.F[v]), "HLLD policies (broken)", i);
        expect(le.code == 0 || sus.any, "a rejected face passes the cheap checks", i);
        rejected += le.code != 0;
        suspected += sus.any;
        if (le.code == 0) {
            double o[14];
            fxo_hlld(WL, WR, pL, pR, g, g, bn, o);
            for (int v = 0; v < 9; ++v) expect(same(a.F[v], o[v]), "HLLD flux", i);
            for (int v = 0; v < 3; ++v) expect(same(a.v[v], o[9 + v]), "HLLD velocity", i);
            expect(same(a.bv1, o[12]) && same(a.bv2, o[13]), "HLLD EMF", i);
        }
        if (!brk) {
            /* the far side's energy and composition are not looked at, but
             * for the HLL fallback, which asks for both sides */
            int asked = 0;
            FxFaceOut c;
            memset(&c, 0, sizeof c);
            double VL[9], VR[9];
            memcpy(VL, WL, sizeof VL);
            memcpy(VR, WR, sizeof VR);
            VL[4] = VL[5] = VR[4] = VR[5] = NAN;
            FxErrLocal lc;
            fx_riemann_hlld_folded_br(VL, VR, pL, pR, g, g, bn, c, &lc, 1, 2, br, [&](bool left, double &eint, double &ye) {
                ++asked;
                eint = left ? WL[4] : WR[4];
                ye = left ? WL[5] : WR[5];
            });
            expect(memcmp(&b, &c, sizeof b) == 0 && lc.code == le.code && asked >= 1, "HLLD near side", i);
            one += asked == 1;
            ++sound;
            doubtful += sus.any;
        }
        double F[6], vf[3], o[9];
        const double du = sym(), dv = sym(), dw = sym();
        fx_riemann_hllc(WL, WR, pL, pR, g, g, du, dv, dw, F, vf);
        fxo_hllc(WL, WR, pL, pR, g, g, du, dv, dw, o);
        for (int v = 0; v < 6; ++v) expect(same(F[v], o[v]), "HLLC flux", i);
        for (int v = 0; v < 3; ++v) expect(same(vf[v], o[6 + v]), "HLLC velocity", i);
    }
    printf("%ld faces, %ld rejected, %ld suspected, %ld of %ld sound ones suspected, %ld differences\n", n, rejected,
        suspected, doubtful, sound, bad);
    return bad == 0 && rejected > n / 100 && doubtful * 1000 < sound && one > sound * 9 / 10 ? 0 : 1;
}
