/*
 * Rounding error of the face's reverse sweep (fornaxamr_b200/csrc/
 * fx_adjoint.cuh): the header compiled twice, in 64-bit doubles and with every
 * double an 80-bit long double, on the same seeded faces.  Prints the mean
 * over the faces of |g64 - g80| / |g80| (2-norms of the 37 adjoints).  Faces
 * whose decisions differ between the two (a tie at round-off) are left out.
 */
#include <math.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

#include <cmath>

#include "../include/fornax_b200.h"

namespace d64 {
#include "fx_adjoint.cuh"
}
#undef FX_ADJOINT_CUH
#undef FX_PHYSICS_CUH
#undef FX_LAYOUT_H
namespace d80 {
#define double long double
#include "fx_adjoint.cuh"
#undef double
}

static uint64_t st = 88172645463325252ULL;
static double uni()
{
    st ^= st << 13;
    st ^= st >> 7;
    st ^= st << 17;
    return (double)(st >> 11) * (1.0 / 9007199254740992.0);
}
static double sym() { return 2.0 * uni() - 1.0; }

int main()
{
    const long n = 200000;
    long used = 0;
    double sum = 0.0, worst = 0.0;
    for (long i = 0; i < n; ++i) {
        double w[36], ob[14], wb[36] = {0}, bn = 0.7 * sym(), bnb = 0.0;
        const double v0 = i % 8 == 0 ? 3.0 * sym() : 0.3 * sym(); /* some faces supersonic */
        const double rho = 0.5 + 1.5 * uni(), e = 0.5 + 2.5 * uni(), b2 = sym(), b3 = sym();
        for (int c = 0; c < 4; ++c) {
            double *x = w + 9 * c;
            x[0] = rho * (1.0 + 0.05 * sym());
            x[1] = v0 + 0.05 * sym();
            x[2] = 0.2 * sym();
            x[3] = 0.2 * sym();
            x[4] = e * (1.0 + 0.05 * sym());
            x[5] = 0.1 + 0.01 * sym();
            x[6] = 0.0;
            x[7] = b2 + 0.05 * sym();
            x[8] = b3 + 0.05 * sym();
        }
        for (double &x : ob) x = sym();
        const double g = 5.0 / 3.0;
        d64::fxa_face_vjp(w, g, bn, ob, wb, bnb);
        long double W[36], O[14], Wb[36] = {0}, Bb = 0.0L;
        for (int q = 0; q < 36; ++q) W[q] = w[q];
        for (int q = 0; q < 14; ++q) O[q] = ob[q];
        d80::fxa_face_vjp(W, g, bn, O, Wb, Bb);
        long double num = 0.0L, den = 0.0L;
        for (int q = 0; q < 36; ++q) {
            num += (wb[q] - Wb[q]) * (wb[q] - Wb[q]);
            den += Wb[q] * Wb[q];
        }
        num += (bnb - Bb) * (bnb - Bb);
        den += Bb * Bb;
        const double err = (double)sqrtl(num / den);
        if (!(err < 1e-9)) continue;
        ++used;
        sum += err;
        worst = err > worst ? err : worst;
    }
    printf("%ld of %ld faces, mean %.4g, largest %.3g\n", used, n, sum / used, worst);
    return 0;
}
