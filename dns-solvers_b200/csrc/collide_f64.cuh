// FP64 collision in the reference's operand order (xcomputations.c:314-342).
// Every translation unit that calls f64_collide must be compiled with
// -fmad=false: the bit-exact parity with the reference depends on no fused
// multiply-add.  Zero terms of the reference's sums (E*f with E == 0) are
// omitted: adding a signed zero to a non-zero partial sum leaves it unchanged.
#pragma once

#include "lattice.cuh"

namespace dnslbm {

// Moments in the reference's summation order (a = 0..18).
__device__ __forceinline__ void f64_moments(const double (&f)[Q], double &dens, double &jx, double &jy, double &jz)
{
    dens = 0.0;
#pragma unroll
    for (int a = 0; a < Q; ++a) dens = dens + f[a];
    jx = 0.0;
    jy = 0.0;
    jz = 0.0;
#pragma unroll
    for (int a = 0; a < Q; ++a) {
        if (lat_ex(a) > 0) jx = jx + f[a];
        if (lat_ex(a) < 0) jx = jx - f[a];
        if (lat_ey(a) > 0) jy = jy + f[a];
        if (lat_ey(a) < 0) jy = jy - f[a];
        if (lat_ez(a) > 0) jz = jz + f[a];
        if (lat_ez(a) < 0) jz = jz - f[a];
    }
}

// e_a . u with the reference's grouping (E0*u0 + E1*u1) + E2*u2.
template <int A>
__device__ __forceinline__ double f64_eu(double u0, double u1, double u2)
{
    constexpr int ex = lat_ex(A), ey = lat_ey(A), ez = lat_ez(A);
    double s = 0.0;
    bool first = true;
    if (ex != 0) { s = ex > 0 ? u0 : -u0; first = false; }
    if (ey != 0) { s = first ? (ey > 0 ? u1 : -u1) : (ey > 0 ? s + u1 : s - u1); first = false; }
    if (ez != 0) { s = first ? (ez > 0 ? u2 : -u2) : (ez > 0 ? s + u2 : s - u2); }
    return s;
}

struct F64Cell {
    double dens, jx, u0, u1, u2;
};

// Population A and its opposite B after the collision.  Rounding is symmetric
// in sign, so e_B . u == -(e_A . u) exactly and the pair shares the products
// of e . u: 3 (e.u), 4.5 (e.u)^2 and 9 (e.u) are computed once.
template <int A>
__device__ __forceinline__ void f64_pair(double (&f)[Q], const F64Cell &c, double v15, const double (&wd)[3], double m3,
                                         double p3, double n3, double omega, double G)
{
    constexpr int B = lat_opp(A), ex = lat_ex(A), cls = lat_wclass(A);
    constexpr double w = cls == 1 ? 1. / 18. : 1. / 36.;
    const double u = f64_eu<A>(c.u0, c.u1, c.u2);
    const double u3 = 3. * u, uu = (4.5 * u) * u;
    const double ta = ((1. + u3) + uu) - v15, tb = ((1. - u3) + uu) - v15;
    double bra = m3, brb = m3;
    if (ex != 0) {
        const double u9 = 9. * u;
        bra = ex > 0 ? p3 + u9 : n3 - u9;
        brb = ex > 0 ? n3 + u9 : p3 - u9;
    }
    const double Fa = (w * bra) * G, Fb = ex != 0 ? (w * brb) * G : Fa;
    f[A] = f[A] + (Fa - omega * (f[A] - wd[cls] * ta));
    f[B] = f[B] + (Fb - omega * (f[B] - wd[cls] * tb));
}

// BGK collision with the reference's forcing term, in place.
__device__ __forceinline__ F64Cell f64_collide(double (&f)[Q], double omega, double G)
{
    F64Cell c;
    double jy, jz;
    f64_moments(f, c.dens, c.jx, jy, jz);
    c.u0 = c.jx / c.dens;
    c.u1 = jy / c.dens;
    c.u2 = jz / c.dens;
    const double v15 = 1.5 * (c.u0 * c.u0 + c.u1 * c.u1 + c.u2 * c.u2);
    const double wd[3] = {(1. / 3.) * c.dens, (1. / 18.) * c.dens, (1. / 36.) * c.dens};
    const double m3 = 3. * (0. - c.u0), p3 = 3. * (1. - c.u0), n3 = 3. * (-1. - c.u0);
    // rest direction: e . u = 0
    f[0] = f[0] + (((1. / 3.) * m3) * G - omega * (f[0] - wd[0] * (1. - v15)));
#define DNSLBM_PAIR(A) f64_pair<A>(f, c, v15, wd, m3, p3, n3, omega, G);
    DNSLBM_PAIR(1) DNSLBM_PAIR(3) DNSLBM_PAIR(5) DNSLBM_PAIR(7) DNSLBM_PAIR(8) DNSLBM_PAIR(11) DNSLBM_PAIR(12)
    DNSLBM_PAIR(15) DNSLBM_PAIR(16)
#undef DNSLBM_PAIR
    return c;
}

}  // namespace dnslbm
