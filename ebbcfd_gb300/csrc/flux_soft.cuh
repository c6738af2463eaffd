// flux_soft.cuh -- the plain FP64 face fluxes (source/flux.d) with their quotients,
// square roots and most products on the integer pipe (softdbl.h), bit for bit those of
// device_math.cuh.
//
// The plain FP64 flux kernel is bound by the FP64 pipe (a warp instruction every 64
// cycles of a scheduler: ~440 of them per face kept it 85% busy with 8% of the issue
// slots used).  Here about 125 remain per face, additions mostly, beside ~6,000 other
// instructions: the pipe is 72% busy, the integer pipe 57% (1M plate cells).  Per launch,
// 400,000 plate cells: 195 us, 548 us with device_math.cuh; 200,000 triangles (Rusanov): 40
// and 136 us (both with the boundary faces' part, which used to run last and alone: k_flux).
// Three things keep the integer part from costing what it saves:
//  * code size: as straight-line code a quarter of the warps' time went to instruction
//    fetches (287 us).  The two sides of a face, the two directions of the viscous
//    matrices and the three wave speeds are loops (16% of the time still);
//  * halvings: x/2 is exact, so a halved term is left doubled until it meets an addition,
//    which takes it as a fused multiply-add by 0.5 (one rounding, the same), and the
//    flux itself is returned doubled (the caller halves the edge length instead);
//  * range checks: products need normal operands and results.  With the face states in
//    2^+-60 (density) and 2^+-100 or zero, normals in [2^-100, 2] and (viscous) gradients,
//    viscosity and Prandtl-number terms in 2^+-100, every operand below stays a normal number or an exact
//    zero: a sum of two terms is zero or at least the smaller one's last place, so each
//    sum lowers a bound by 53 binary digits at most, and no chain of products here comes
//    below 2^-960 or above 2^960.  Only the wave strengths C1, C2, which multiply four
//    such factors, are checked where they arise.
// `bad` (never cleared) says that the face has to be evaluated by device_math.cuh.
#pragma once

#include "device_math.cuh"
#include "softdbl.h"

namespace ebbdev {

// S: products on the integer pipe; else on the FP64 pipe (a third of the code: boundary faces)
template <bool S> __device__ __forceinline__ double sm(double a, double b)
{
    if constexpr (S)
        return ebbsoft::mul(a, b);
    else
        return a * b;
}
// the same for an a that is not zero
template <bool S> __device__ __forceinline__ double smn(double a, double b)
{
    if constexpr (S)
        return ebbsoft::mul<true>(a, b);
    else
        return a * b;
}
__device__ __forceinline__ double soft_ratio(double a, double b, bool &bad)
{
    bad |= !ebbsoft::divisor_ok(b);
    return ebbsoft::div(a, ebbsoft::recip(b));
}

// one side of a face: velocity, momentum, pressure, enthalpy and the convective flux
// along the normal (source/flux.d:19-24)
struct SoftSide {
    double rho, u, v, rv0, rv1, p, h;
    ebbsoft::Recip R;
};
template <bool H, bool S>
__device__ __forceinline__ void soft_side(const double q[4], double nx, double ny, SoftSide &o, double f[4], bool &bad)
{
    const double rho = q[0], e = q[3];
    ebbsoft::check<60>(rho, bad);
    bad |= !(ebbsoft::hi_of(rho) < 0x7ff00000u) || ebbsoft::hi_of(rho) == 0u;  // positive
#pragma unroll
    for (int k = 1; k < 4; k++) ebbsoft::check<100>(q[k], bad);
    o.rho = rho;
    o.R = ebbsoft::recip(rho);
    const double u = ebbsoft::div(q[1], o.R), v = ebbsoft::div(q[2], o.R);
    o.u = u;
    o.v = v;
    const double uu = sm<S>(u, u), vv = sm<S>(v, v);
    o.rv0 = smn<S>(rho, u);
    o.rv1 = smn<S>(rho, v);
    const double p = smn<S>(K<double>::gm1, fma(-0.5, smn<S>(rho, uu + vv), e));
    o.p = p;
    const double pe = p + e;
    if (H) o.h = ebbsoft::div(pe, o.R);
    const double f1 = p + smn<S>(rho, uu), f2 = sm<S>(o.rv0, v), f3 = sm<S>(u, pe);
    const double h2 = p + smn<S>(rho, vv), h3 = sm<S>(v, pe);
    f[0] = sm<S>(o.rv0, nx) + sm<S>(o.rv1, ny);
    f[1] = sm<S>(f1, nx) + sm<S>(f2, ny);
    f[2] = sm<S>(f2, nx) + sm<S>(h2, ny);
    f[3] = sm<S>(f3, nx) + sm<S>(h3, ny);
}

// both sides in one loop: A and B, and the sum of their convective fluxes
template <bool H, bool S>
__device__ __forceinline__ void soft_sides(const double qL[4], const double qR[4], double nx, double ny, SoftSide &A,
                                           SoftSide &B, double fs[4], bool &bad)
{
    double fp[4];
    B = {};
    fs[0] = fs[1] = fs[2] = fs[3] = 0.0;
#pragma unroll 1
    for (int s = 0; s < 2; s++) {
        double q[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            q[k] = s ? qR[k] : qL[k];
            fp[k] = fs[k];
        }
        A = B;
        soft_side<H, S>(q, nx, ny, B, fs, bad);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) fs[k] = fp[k] + fs[k];
}

// the entropy-fixed wave speeds |u + a|, |u - a|, |u| (l1, l2, l3)
__device__ __forceinline__ void soft_speeds(double u, double a, double &l1, double &l2, double &l3, bool &bad)
{
    const double eps = ebbsoft::mul<true>(0.01, a);
    l1 = fabs(u + a);
    l2 = fabs(u - a);
    l3 = fabs(u);
    if (l1 < eps || l2 < eps || l3 < eps) {
        const double e2 = ebbsoft::mul<true>(eps, eps), d = ebbsoft::twice(eps);
        bad |= !ebbsoft::divisor_ok(d);
        const ebbsoft::Recip R = ebbsoft::recip(d);
#pragma unroll 1
        for (int r = 0; r < 3; r++) {
            const double l = l1 < eps ? ebbsoft::div(e2 + ebbsoft::mul(l1, l1), R) : l1;
            l1 = l2;
            l2 = l3;
            l3 = l;
        }
    }
}

// twice the Roe flux (source/flux.d:224-303)
template <bool S>
__device__ __forceinline__ void roe_flux2_soft(const double qL[4], const double qR[4], double nx, double ny, double out[4],
                                               double &sMax, bool &bad)
{
    SoftSide A, B;
    double fs[4];
    soft_sides<true, S>(qL, qR, nx, ny, A, B, fs, bad);
    const double di = ebbsoft::root(ebbsoft::div(B.rho, A.R), bad);
    const double d1 = soft_ratio(1.0, 1.0 + di, bad);
    const double vel0 = smn<S>(d1, smn<S>(di, B.u) + A.u);
    const double vel1 = smn<S>(d1, smn<S>(di, B.v) + A.v);
    const double u = sm<S>(vel0, nx) + sm<S>(vel1, ny);
    const double h = smn<S>(d1, smn<S>(di, B.h) + A.h);
    const double vv = sm<S>(vel0, vel0) + sm<S>(vel1, vel1);
    const double a = ebbsoft::root(smn<S>(K<double>::gm1d, fma(-0.5, vv, h)), bad);
    bad |= !ebbsoft::divisor_ok(a);
    const double dRV0 = B.rv0 - A.rv0, dRV1 = B.rv1 - A.rv1;
    const double dRho = qR[0] - qL[0], dRhoE = qR[3] - qL[3];
    double l1, l2, l3;
    soft_speeds(u, a, l1, l2, l3, bad);
    sMax = max4(l1, l2, l3, l3);
    // s1 - l3 and twice s2; G1's first term doubled
    const double sl = fma(0.5, l1 + l2, -l3), s2 = l1 - l2;
    const double qq = ebbsoft::root(vv, bad);
    const double G1 = smn<S>(K<double>::gm1, fma(0.5, sm<S>(sm<S>(qq, qq), dRho), -(sm<S>(vel0, dRV0) + sm<S>(vel1, dRV1))) + dRhoE);
    const double G2 = sm<S>(-u, dRho) + (sm<S>(dRV0, nx) + sm<S>(dRV1, ny));
    const ebbsoft::Recip R = ebbsoft::recip(a);
    const double C1 = fma(0.5, ebbsoft::div(G2, R) * s2, soft_ratio(G1, ebbsoft::mul<true>(a, a), bad) * sl);
    const double C2 = fma(0.5, ebbsoft::div(G1, R) * s2, sl * G2);
    ebbsoft::check<400>(C1, bad);
    ebbsoft::check<400>(C2, bad);
    out[0] = fs[0] - (smn<S>(l3, dRho) + C1);
    out[1] = fs[1] - (smn<S>(l3, dRV0) + sm<S>(C1, vel0) + sm<S>(C2, nx));
    out[2] = fs[2] - (smn<S>(l3, dRV1) + sm<S>(C1, vel1) + sm<S>(C2, ny));
    out[3] = fs[3] - (smn<S>(l3, dRhoE) + sm<S>(C1, h) + sm<S>(C2, u));
}

// twice the Rusanov flux (source/flux.d:66-141, the reduced form of rusanov_flux)
template <bool S>
__device__ __forceinline__ void rusanov_flux2_soft(const double qL[4], const double qR[4], double nx, double ny,
                                                   double out[4], double &sMax, bool &bad)
{
    SoftSide A, B;
    double fs[4];
    soft_sides<false, S>(qL, qR, nx, ny, A, B, fs, bad);
    const double rho = ebbsoft::root(smn<S>(A.rho, B.rho), bad);
    const double sL = ebbsoft::root(A.rho, bad), sR = ebbsoft::root(B.rho, bad);
    const ebbsoft::Recip D = ebbsoft::recip(sL + sR);
    const double vel0 = ebbsoft::div(smn<S>(sL, A.u) + smn<S>(sR, B.u), D);
    const double vel1 = ebbsoft::div(smn<S>(sL, A.v) + smn<S>(sR, B.v), D);
    const double u = sm<S>(vel0, nx) + sm<S>(vel1, ny);
    const double p = ebbsoft::div(smn<S>(sL, A.p) + smn<S>(sR, B.p), D);
    const double a = ebbsoft::root(smn<S>(K<double>::g, ebbsoft::div(p, ebbsoft::recip(rho))), bad);
    bad |= !ebbsoft::divisor_ok(a);
    double l1, l2, l3;
    soft_speeds(u, a, l1, l2, l3, bad);
    const double s = max4(l1, l2, l3, l3);
    sMax = s;
    out[0] = fs[0] - smn<S>(s, qR[0] - qL[0]);
    out[1] = fs[1] - smn<S>(s, B.rv0 - A.rv0);
    out[2] = fs[2] - smn<S>(s, B.rv1 - A.rv1);
    out[3] = fs[3] - smn<S>(s, qR[3] - qL[3]);
}

template <bool S>
__device__ __forceinline__ void inviscid_flux2_soft(int kind, const double qL[4], const double qR[4], double nx, double ny,
                                                    double out[4], double &sMax, bool &bad)
{
    if (kind == 1)
        roe_flux2_soft<S>(qL, qR, nx, ny, out, sMax, bad);
    else
        rusanov_flux2_soft<S>(qL, qR, nx, ny, out, sMax, bad);
}

// Twice the viscous flux (source/flux.d:28-64) of the face state q and gradients dq, or of
// their halves: the quotients by the density do not see a factor in q, mu over the density
// takes it on, and the fluxes are linear in dq.  Component 0 is a signed zero (zero_dot) and
// left to the caller.  Directions x and y run the same loop body: a matrix entry of the
// second is the first's with u and v (and the two coefficients of a pair) exchanged.
template <bool S>
__device__ __forceinline__ void diffusive_flux2_soft(const ViscConst<double> &vc, double mu, const double q[4],
                                                     const double dq[4][2], double nx, double ny, double out[4], bool &bad)
{
    ebbsoft::check<100>(mu, bad);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        ebbsoft::check<100>(dq[k][0], bad);
        ebbsoft::check<100>(dq[k][1], bad);
    }
    const ebbsoft::Recip R = ebbsoft::recip(q[0]);
    const double u = ebbsoft::div(q[1], R), v = ebbsoft::div(q[2], R), E = ebbsoft::div(q[3], R);
    bad |= (ebbsoft::hi_of(mu) & ebbsoft::kExp) == 0u;
    const double s = ebbsoft::div(ebbsoft::twice(mu), R);
    const double c43 = -4.0 / 3.0, p43 = 4.0 / 3.0, m23 = -2.0 / 3.0, c231 = 2.0 / 3.0 - 1.0;
    const double uu = sm<S>(u, u), vv = sm<S>(v, v), gE = smn<S>(vc.gP, E);
    const double b30 = smn<S>(s, sm<S>(smn<S>(c231, u), v));
    const double sp43 = smn<S>(s, p43), sm23 = smn<S>(s, m23), sgP = smn<S>(s, vc.gP);
    const double su = smn<S>(s, u), sv = smn<S>(s, v), tu = smn<S>(s, smn<S>(m23, u)), tv = smn<S>(s, smn<S>(m23, v));
    // row 2 of the x matrices is row 1 of the y ones
    const double G12 = (zero_plus(sm<S>(-sv, dq[0][0])) + smn<S>(s, dq[2][0])) +
                       (zero_plus(sm<S>(-su, dq[0][1])) + smn<S>(s, dq[1][1]));
    double Gn[4];  // G0_1, G0_3, G1_2, G1_3
    double z0 = dq[0][0], z1 = dq[1][0], z2 = dq[2][0], z3 = dq[3][0];
    double w0 = dq[0][1], w1 = dq[1][1], w2 = dq[2][1], w3 = dq[3][1];
    double zn = z1;                                // normal-stress gradient
    double U = u, tV = -tv, tW = -tu;              // velocity along; s 2/3 times that across
    double tA = vc.c43gP, tB = vc.m1gP, kA = vc.p43mgP, kB = vc.omgP, eA = sv, eB = tu;
    auto next_direction = [&]() {
        zn = w2;
        double x = z0;
        z0 = w0, w0 = x;
        x = z1, z1 = w1, w1 = x;
        x = z2, z2 = w2, w2 = x;
        z3 = w3;
        U = v;
        tV = tW;
        x = tA, tA = tB, tB = x;
        x = kA, kA = kB, kB = x;
        eA = tv;
        eB = su;
    };
    auto rows = [&](double &n, double &e) {
        n = (zero_plus(sm<S>(smn<S>(s, smn<S>(c43, U)), z0)) + smn<S>(sp43, zn)) +
            (zero_plus(sm<S>(tV, w0)) + smn<S>(sm23, w2));
        const double t = sm<S>(tA, uu) + sm<S>(tB, vv) - gE;
        e = (zero_plus(sm<S>(smn<S>(s, t), z0)) + sm<S>(smn<S>(s, sm<S>(kA, u)), z1) +
             sm<S>(smn<S>(s, sm<S>(kB, v)), z2) + smn<S>(sgP, z3)) +
            (zero_plus(sm<S>(b30, w0)) + sm<S>(eA, w1) + sm<S>(eB, w2));
    };
#pragma unroll 1
    for (int d = 0; d < 2; d++) {
        Gn[0] = Gn[2];
        Gn[1] = Gn[3];
        rows(Gn[2], Gn[3]);
        next_direction();
    }
    out[1] = sm<S>(Gn[0], nx) + sm<S>(G12, ny);
    out[2] = sm<S>(G12, nx) + sm<S>(Gn[2], ny);
    out[3] = sm<S>(Gn[1], nx) + sm<S>(Gn[3], ny);
}

}  // namespace ebbdev
