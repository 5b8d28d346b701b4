// numerics_nr.cuh — the face flux of the exact build with correctly rounded
// FP64 division in straight-line code.
//
// The compiler's division is correctly rounded, but each one ends in a range
// test with a branch to a slow path.  A face has 106 of them: they were half
// of its instructions, and their branches split the flux into short pieces
// that the scheduler cannot interleave, so the FP64 pipe idled half of the
// time on dependent chains.  DivNR forms the same quotients, bit for bit:
//
//  - Reciprocal: the hardware approximation (PTX rcp.approx.ftz.f64, relative
//    error below 2^-19.9: it reads the upper word of b) refined by two
//    Newton-Raphson steps, e = 1 - b*y, y = y + y*e.  Each squares the error,
//    so y is the rounding of (1/b)(1 + h) with |h| < 2^-79, and
//    |b*y - 1| <= b u (1 + 2^-24) with b scaled to [1, 2) and u = 2^-54, half
//    an ulp of y.
//  - Quotient: q0 = a*y, q1 = q0 + (a - b*q0)*y by two FMAs.  q1 is RN(a/b):
//    what is rounded is a/b + (a/b - q0)(b*y - 1), so q1 can be wrong only
//    when a/b lies closer to the midpoint M of two doubles than that second
//    term.  Then a*y is less than an ulp from M, so q0 is one of M's two
//    neighbours and the term is at most half an ulp times b u (1 + 2^-24);
//    but a/b is no midpoint (a 53-bit b times a 54-bit M is no 53-bit a), and
//    a - b*M is a multiple of 2^-106 (a/b < 1) or 2^-105, so |a/b - M| is at
//    least 2 u / b of an ulp.  That is the larger one while
//    b^2 (1 + 2^-24) < 4: for every b whose upper 24 fraction bits are not all
//    ones.  (The argument is Markstein's, for y = RN(1/b): IBM J. Res. Dev.
//    34(1), 1990; it holds for the constant denominators with y = RN(1/b)
//    from the host whatever their bits.)
//  - eps + IS2 has those bits all ones often: IS2 rounds to minus a power of
//    two where the data is nearly constant.  A third Newton-Raphson step
//    makes y = RN(1/b) there, and so every b good: with b j ulps below 2, 1/b
//    is at least j^2 2^-106 (relative) from a midpoint for odd j and further
//    for even j, and the step errs by 2^-104 at most.  Only j = 1, every bit a
//    one, needs care: from y = 1/2 the step lands on a tie, which the lowest
//    bit set in the factor y of the correction breaks upwards, to RN(1/b).
//
// Denominators with those bits all ones, or outside the ranges below, and
// numerators so small that a remainder could be inexact clear ok, and the
// face is computed again with the compiler's division.  A zero numerator is
// exact.  The smoothness ratio tau/(eps + IS) only enters 1 + ratio, where a
// ratio below 2^-60 vanishes however it was rounded, and a ratio that
// overflows shows in the sum of the weights, whose range is tested: tau
// needs no test of its own.
#pragma once
#include "numerics.cuh"

namespace fdm {

// a denominator and its reciprocal, rounded as the text above says; DenC:
// exactly RN(1/b)
struct Den {
    double b, y;
};
struct DenC {
    double b, y;
};
// the constant denominators with their reciprocals (IEEE division on the
// host); passed to kernels by value
struct FluxDen {
    DenC gm1, d2;
};
inline FluxDen flux_den(double g) {
    return FluxDen{DenC{g - 1.0, 1.0 / (g - 1.0)}, DenC{FDM_D2_WCNS, 1.0 / FDM_D2_WCNS}};
}

struct DivNR {
    DenC gm1, d2;    // constant denominators, y = RN(1/b) from the host
    bool ok = true;

    __device__ __forceinline__ explicit DivNR(const FluxDen &c) : gm1(c.gm1), d2(c.d2) {}

    // upper word of |x|
    __device__ __forceinline__ static unsigned hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
    // the upper 24 fraction bits are not all ones
    __device__ __forceinline__ void test_bits(double b) {
        ok = ok && __funnelshift_l((unsigned)__double2loint(b), (unsigned)__double2hiint(b), 12) < 0xffffff00u;
    }
    // 2^LO <= |b| < 2^HI (NaN and infinity fail)
    template <int LO, int HI>
    __device__ __forceinline__ void test_range(double b) {
        ok = ok && hi(b) - ((unsigned)(1023 + LO) << 20) < ((unsigned)(HI - LO) << 20);
    }
    // zero or at least 2^-800
    __device__ __forceinline__ void test_numerator(double a) {
        const unsigned k = hi(a) | min((unsigned)__double2loint(a), 1u);
        ok = ok && k - 1u >= ((unsigned)(1023 - 800) << 20) - 1u;
    }
    __device__ __forceinline__ static Den den(double b) {
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
        double e = __fma_rn(-b, y, 1.0);
        y = __fma_rn(y, e, y);
        e = __fma_rn(-b, y, 1.0);
        return Den{b, __fma_rn(y, e, y)};
    }
    __device__ __forceinline__ static Den den3(double b) {
        const double y = den(b).y;
        const double odd = __hiloint2double(__double2hiint(y), __double2loint(y) | 1);
        return Den{b, __fma_rn(odd, __fma_rn(-b, y, 1.0), y)};
    }
    __device__ __forceinline__ static double q(double a, double b, double y) {
        const double q0 = a * y;
        return __fma_rn(__fma_rn(-b, q0, a), y, q0);
    }
    __device__ __forceinline__ static double q(double a, const Den &d) { return q(a, d.b, d.y); }
    __device__ __forceinline__ static double q(double a, const DenC &d) { return q(a, d.b, d.y); }
};
// the same interface with the compiler's division
struct DivIEEE {
    DenC gm1, d2;
    static constexpr bool ok = true;
    __device__ __forceinline__ explicit DivIEEE(const FluxDen &c) : gm1(c.gm1), d2(c.d2) {}
    __device__ __forceinline__ void test_bits(double) {}
    template <int LO, int HI>
    __device__ __forceinline__ void test_range(double) {}
    __device__ __forceinline__ void test_numerator(double) {}
    __device__ __forceinline__ static Den den(double b) { return Den{b, 0.0}; }
    __device__ __forceinline__ static double q(double a, const Den &d) { return a / d.b; }
    __device__ __forceinline__ static double q(double a, const DenC &d) { return a / d.b; }
};

// The characteristic basis of a face (eigen) in the few quotients that
// differ: with the momentum columns named by their direction (n the face's,
// t along it), Ri(1,t) = -2 Ri(0,t), Ri(2,t) = Ri(0,t) and the same in the
// energy column, exactly (the denominators are a*a and 2*a*a, the numerators
// differ in sign).
struct EigNR {
    double u, v, a, q2, H1, H2;
    double R00, R10, R20;   // column 0
    double R0n, R1n, R2n;   // the face's own momentum column
    double Ct, C3;          // Ri(0,t), Ri(0,3)
};
template <int DIR>
__device__ __forceinline__ void eigen_nr(const double Um[4], double g, DivNR &dv, EigNR &E) {
    const double r0 = Um[0];
    dv.test_bits(r0);
    dv.test_range<-100, 100>(r0);
    dv.test_numerator(Um[1]);
    dv.test_numerator(Um[2]);
    const Den dr = DivNR::den(r0);
    const double u = DivNR::q(Um[1], dr), v = DivNR::q(Um[2], dr);
    const double p = (g - 1.0) * r0 * (DivNR::q(Um[3], dr) - 0.5 * (u * u + v * v));
    const double a = sqrt(DivNR::q(g * p, dr));
    const double q2 = 0.5 * (u * u + v * v);
    const double aa = a * a;
    dv.test_bits(aa);
    dv.test_range<-100, 100>(aa);   // a tiny, zero or negative p shows here
    const Den daa = DivNR::den(aa), da2{2.0 * aa, 0.5 * daa.y};
    const double c = DIR == 0 ? u : v, t = DIR == 0 ? v : u;
    E.u = u; E.v = v; E.a = a; E.q2 = q2;
    const double h = DivNR::q(aa, dv.gm1) + q2;
    E.H1 = h - c * a;
    E.H2 = h + c * a;
    E.R00 = DivNR::q((g - 1.0) * q2 + a * c, da2);
    E.R10 = DivNR::q(aa - (g - 1.0) * q2, daa);
    E.R20 = DivNR::q((g - 1.0) * q2 - a * c, da2);
    E.R0n = DivNR::q((1.0 - g) * c - a, da2);
    E.R1n = DivNR::q((g - 1.0) * c, daa);
    E.R2n = DivNR::q((1.0 - g) * c + a, da2);
    E.Ct = DivNR::q((1.0 - g) * t, da2);
    E.C3 = DivNR::q(g - 1.0, da2);
}
// w = Ri * X in MATMUL order; the products with the shared entries are
// formed once, and -2 times such a product is exact
template <int DIR>
__device__ __forceinline__ void project_nr(const EigNR &E, const double X[4], double w[4]) {
    const double h3 = E.C3 * X[3];
    if (DIR == 0) {
        const double h2 = E.Ct * X[2];
        w[0] = E.R00 * X[0] + E.R0n * X[1] + h2 + h3;
        w[1] = __fma_rn(-2.0, h3, __fma_rn(-2.0, h2, E.R10 * X[0] + E.R1n * X[1]));
        w[2] = E.R20 * X[0] + E.R2n * X[1] + h2 + h3;
        w[3] = E.v * X[0] + -X[2];
    } else {
        const double h1 = E.Ct * X[1];
        w[0] = E.R00 * X[0] + h1 + E.R0n * X[2] + h3;
        w[1] = __fma_rn(-2.0, h3, __fma_rn(-2.0, h1, E.R10 * X[0]) + E.R1n * X[2]);
        w[2] = E.R20 * X[0] + h1 + E.R2n * X[2] + h3;
        w[3] = -E.u * X[0] + X[1];
    }
}
template <int DIR>
__device__ __forceinline__ void back_project_nr(const EigNR &E, const double uL[4], double hp[4]) {
    hp[0] = uL[0] + uL[1] + uL[2];
    if (DIR == 0) {
        hp[1] = (E.u - E.a) * uL[0] + E.u * uL[1] + (E.u + E.a) * uL[2];
        hp[2] = E.v * uL[0] + E.v * uL[1] + E.v * uL[2] + -uL[3];
        hp[3] = E.H1 * uL[0] + E.q2 * uL[1] + E.H2 * uL[2] + -E.v * uL[3];
    } else {
        hp[1] = E.u * uL[0] + E.u * uL[1] + E.u * uL[2] + uL[3];
        hp[2] = (E.v - E.a) * uL[0] + E.v * uL[1] + (E.v + E.a) * uL[2];
        hp[3] = E.H1 * uL[0] + E.q2 * uL[1] + E.H2 * uL[2] + E.u * uL[3];
    }
}
// the smaller of two squares (a NaN gives way to the other, as fmin's does)
__device__ __forceinline__ double min_square(double a, double b) {
    const unsigned long long x = (unsigned long long)__double_as_longlong(a), y = (unsigned long long)__double_as_longlong(b);
    return __longlong_as_double((long long)(x < y ? x : y));
}
// the weights' end of wcns_z3: smoothness indicators in, value out
__device__ __forceinline__ double wcns_weigh(double u1, double u2, double u3, double IS1, double IS2, DivNR &dv) {
    const double d1 = FDM_D1_WCNS, d2 = FDM_D2_WCNS;
    double t = 10. * fabs(IS2 - 3. * IS1);
    const double tau3 = t * t;
    const double b1 = FDM_EPS_WCNS + IS1, b2 = FDM_EPS_WCNS + IS2;
    dv.test_bits(b1);
    dv.test_range<-200, 450>(b2);   // IS2 can round to a negative value; IS1 cannot, and IS1 <= IS2 otherwise
    const double a1 = d1 * (1.0 + DivNR::q(tau3, DivNR::den(b1)));
    const double a2 = d2 * (1.0 + DivNR::q(tau3, DivNR::den3(b2)));
    const double s = a1 + a2;
    dv.test_bits(s);
    dv.test_range<-200, 450>(s);
    const Den ds = DivNR::den(s);
    const double x = (-u1 + 6.0 * u2 + 3.0 * u3) / 8.0 - d1 * u2;
    dv.test_numerator(x);
    const double p2 = DivNR::q(x, dv.d2);
    return DivNR::q(a1, ds) * u2 + DivNR::q(a2, ds) * p2;
}
// wcns_z3 of (w0, w1, w2) and of (w3, w2, w1): the squares and the product
// of the two middle values are the same in both, and subtracting 2*u2 (exact)
// is one FMA
__device__ __forceinline__ void wcns_pair(double w0, double w1, double w2, double w3, DivNR &dv, double &L, double &R) {
    double t = w2 - w1;
    const double m2 = t * t, s1 = w1 * w1, s2 = w2 * w2, x12 = w1 * w2;
    t = w1 - w0;
    double IS1 = min_square(t * t, m2);
    t = __fma_rn(-2.0, w1, w0) + w2;
    double IS2 = t * t + w0 * w0 + s1 + s2 - w0 * w1 - x12 - w0 * w2;
    L = wcns_weigh(w0, w1, w2, IS1, IS2, dv);
    t = w2 - w3;
    IS1 = min_square(t * t, m2);
    t = __fma_rn(-2.0, w2, w3) + w1;
    IS2 = t * t + w3 * w3 + s2 + s1 - w3 * w2 - x12 - w3 * w1;
    R = wcns_weigh(w3, w2, w1, IS1, IS2, dv);
}
template <int DIR>
__device__ __forceinline__ void cons_state_nr(const Prim &q, const DivNR &dv, double U[4]) {
    const double ke = q.u * q.u + q.v * q.v;
    U[0] = q.r;
    U[1] = q.r * q.u;
    U[2] = q.r * q.v;
    U[3] = DivNR::q(q.p, dv.gm1) + 0.5 * q.r * ke;
}
template <int DIR, class D>
__device__ __forceinline__ void phys_flux_nr(const Prim &q, const D &dv, double F[4]) {
    const double ke = q.u * q.u + q.v * q.v;
    const double e = D::q(q.p, dv.gm1) + 0.5 * q.r * ke;
    if (DIR == 0) {
        F[0] = q.r * q.u;
        F[1] = q.r * q.u * q.u + q.p;
        F[2] = q.r * q.u * q.v;
        F[3] = q.u * (e + q.p);
    } else {
        F[0] = q.r * q.v;
        F[1] = q.r * q.u * q.v;
        F[2] = q.r * q.v * q.v + q.p;
        F[3] = q.v * (e + q.p);
    }
}

// face_flux_slots (numerics.cuh) with DivNR: the state half,
// then the flux half from the records read again; the values of the face are
// wrong when dv.ok is false afterwards.
template <int DIR>
__device__ __forceinline__ void face_flux_nr(const double4 *__restrict__ cur, int32_t ia, int32_t ib, int32_t ic,
                                             int32_t id, double g, DivNR &dv, double lam, double out[4]) {
    double wL[4], wR[4];
    EigNR E;
    {
        const Prim s0 = load_prim(cur, ia), s1 = load_prim(cur, ib), s2 = load_prim(cur, ic), s3 = load_prim(cur, id);
        dv.test_numerator(s0.p);
        dv.test_numerator(s1.p);
        dv.test_numerator(s2.p);
        dv.test_numerator(s3.p);
        double U0[4], U1[4], U2[4], U3[4];
        cons_state_nr<DIR>(s1, dv, U1);
        cons_state_nr<DIR>(s2, dv, U2);
        double Um[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) Um[r] = (U1[r] + U2[r]) / 2.0;
        eigen_nr<DIR>(Um, g, dv, E);
        cons_state_nr<DIR>(s0, dv, U0);
        cons_state_nr<DIR>(s3, dv, U3);
        double w0[4], w1[4], w2[4], w3[4], uwL[4], uwR[4];
        project_nr<DIR>(E, U0, w0); project_nr<DIR>(E, U1, w1);
        project_nr<DIR>(E, U2, w2); project_nr<DIR>(E, U3, w3);
#pragma unroll
        for (int r = 0; r < 4; ++r) wcns_pair(w0[r], w1[r], w2[r], w3[r], dv, uwL[r], uwR[r]);
        back_project_nr<DIR>(E, uwL, wL);
        back_project_nr<DIR>(E, uwR, wR);
    }
    double F0[4], F1[4], F2[4], F3[4];
    phys_flux_nr<DIR>(load_prim(cur, ia), dv, F0);
    phys_flux_nr<DIR>(load_prim(cur, ib), dv, F1);
    phys_flux_nr<DIR>(load_prim(cur, ic), dv, F2);
    phys_flux_nr<DIR>(load_prim(cur, id), dv, F3);
    double w0[4], w1[4], w2[4], w3[4], ugL[4], ugR[4];
    project_nr<DIR>(E, F0, w0); project_nr<DIR>(E, F1, w1);
    project_nr<DIR>(E, F2, w2); project_nr<DIR>(E, F3, w3);
#pragma unroll
    for (int r = 0; r < 4; ++r) wcns_pair(w0[r], w1[r], w2[r], w3[r], dv, ugL[r], ugR[r]);
    double gL[4], gR[4];
    back_project_nr<DIR>(E, ugL, gL);
    back_project_nr<DIR>(E, ugR, gR);
#pragma unroll
    for (int r = 0; r < 4; ++r) out[r] = 0.5 * (gL[r] + gR[r] - lam * (wR[r] - wL[r]));
}
// a face that DivNR refuses, out of line: the compiler's division
template <int DIR>
__device__ __noinline__ double4 face_flux_again(const double4 *cur, int32_t ia, int32_t ib, int32_t ic, int32_t id,
                                                double g, double lam) {
    double out[4];
    face_flux_slots<DIR>(cur, ia, ib, ic, id, g, lam, out);
    return make_double4(out[0], out[1], out[2], out[3]);
}
// the flux of the face with stencil slots a, b, c, d
template <int DIR>
__device__ __forceinline__ double4 face_flux_of(const double4 *__restrict__ cur, int32_t a, int32_t b, int32_t c,
                                                int32_t d, double g, const FluxDen &den, double lam) {
    double out[4];
    DivNR dv(den);
    face_flux_nr<DIR>(cur, a, b, c, d, g, dv, lam, out);
    return dv.ok ? make_double4(out[0], out[1], out[2], out[3]) : face_flux_again<DIR>(cur, a, b, c, d, g, lam);
}


// one half's values of a point: the conserved state or the physical flux
template <int DIR>
__device__ __forceinline__ void point_half_nr(const Prim &q, const DivNR &dv, bool flux, double X[4]) {
    const double ke = q.u * q.u + q.v * q.v;
    const double e = DivNR::q(q.p, dv.gm1) + 0.5 * q.r * ke;
    const double ru = q.r * q.u, rv = q.r * q.v;
    if (DIR == 0) {
        X[0] = flux ? ru : q.r;
        X[1] = flux ? ru * q.u + q.p : ru;
        X[2] = flux ? ru * q.v : rv;
        X[3] = flux ? q.u * (e + q.p) : e;
    } else {
        X[0] = flux ? rv : q.r;
        X[1] = flux ? ru * q.v : ru;
        X[2] = flux ? rv * q.v + q.p : rv;
        X[3] = flux ? q.v * (e + q.p) : e;
    }
}
// The same flux by two neighbouring lanes: lane bit 0 takes the state half or
// the flux half, which run one code, and ends with components 0 and 1 or 2 and
// 3; only the face's basis is computed twice.  All lanes of the warp call it.
template <int DIR>
__device__ __forceinline__ double2 face_flux_pair(const double4 *__restrict__ cur, int32_t a, int32_t b, int32_t c,
                                                  int32_t d, double g, const FluxDen &den, double lam) {
    const bool flux = threadIdx.x & 1;
    DivNR dv(den);
    double T[4];
    {
        const Prim s0 = load_prim(cur, a), s1 = load_prim(cur, b), s2 = load_prim(cur, c), s3 = load_prim(cur, d);
        dv.test_numerator(s0.p);
        dv.test_numerator(s1.p);
        dv.test_numerator(s2.p);
        dv.test_numerator(s3.p);
        double U1[4], U2[4], Um[4];
        cons_state_nr<DIR>(s1, dv, U1);
        cons_state_nr<DIR>(s2, dv, U2);
#pragma unroll
        for (int r = 0; r < 4; ++r) Um[r] = (U1[r] + U2[r]) / 2.0;
        EigNR E;
        eigen_nr<DIR>(Um, g, dv, E);
        double X[4], w0[4], w1[4], w2[4], w3[4], uL[4], uR[4], L[4], R[4];
        point_half_nr<DIR>(s0, dv, flux, X); project_nr<DIR>(E, X, w0);
        point_half_nr<DIR>(s1, dv, flux, X); project_nr<DIR>(E, X, w1);
        point_half_nr<DIR>(s2, dv, flux, X); project_nr<DIR>(E, X, w2);
        point_half_nr<DIR>(s3, dv, flux, X); project_nr<DIR>(E, X, w3);
#pragma unroll
        for (int r = 0; r < 4; ++r) wcns_pair(w0[r], w1[r], w2[r], w3[r], dv, uL[r], uR[r]);
        back_project_nr<DIR>(E, uL, L);
        back_project_nr<DIR>(E, uR, R);
#pragma unroll
        for (int r = 0; r < 4; ++r) T[r] = R[r] + (flux ? L[r] : -L[r]);
    }
    const bool ok = __shfl_xor_sync(0xffffffffu, (int)dv.ok, 1) && dv.ok;
    double o[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const double got = __shfl_xor_sync(0xffffffffu, flux ? T[r] : T[2 + r], 1);
        const double sum = flux ? T[2 + r] : got, dif = flux ? got : T[r];
        o[r] = 0.5 * (sum - lam * dif);
    }
    if (!ok) {
        const double4 f = face_flux_again<DIR>(cur, a, b, c, d, g, lam);
        o[0] = flux ? f.z : f.x;
        o[1] = flux ? f.w : f.y;
    }
    return make_double2(o[0], o[1]);
}

}  // namespace fdm
