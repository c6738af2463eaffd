// flux_df.cuh -- the double-float face fluxes (source/flux.d) on pairs of double-floats
// (dfpair.cuh): device_math.cuh's expressions with the two sides of a face, the two
// directions or two components in each packed operation.
#pragma once

#include "device_math.cuh"
#include "dfpair.cuh"

namespace ebbdev {

// velocity, momentum, pressure, enthalpy of the two sides (left, right)
struct DfSides {
    dfp rho, u, v, rv0, rv1, p, h, r;  // r: 1 / rho
};
// and the sums over the sides of their convective fluxes, components (0, 3) and (1, 2)
__device__ __forceinline__ void df_sides(const df qL[4], const df qR[4], df nx, df ny, DfSides &S, dfp &f03, dfp &f12)
{
    const dfp e = pair(qL[3], qR[3]), m0 = pair(qL[1], qR[1]), m1 = pair(qL[2], qR[2]);
    S.rho = pair(qL[0], qR[0]);
    S.r = recip(S.rho);
    S.u = m0 * S.r;
    S.v = m1 * S.r;
    S.rv0 = S.rho * S.u;
    S.rv1 = S.rho * S.v;
    const dfp uu = S.u * S.u, vv = S.v * S.v;
    S.p = both(K<df>::gm1) * (e - half(S.rho) * (uu + vv));
    const dfp pe = S.p + e, x = both(nx), y = both(ny);
    S.h = pe * S.r;
    const dfp g2 = S.rv0 * S.v;
    const dfp f0 = S.rv0 * x + S.rv1 * y, f1 = (S.p + S.rho * uu) * x + g2 * y, f2 = g2 * x + (S.p + S.rho * vv) * y,
              f3 = (S.u * pe) * x + (S.v * pe) * y;
    f03 = pair(first(f0), first(f3)) + pair(second(f0), second(f3));
    f12 = pair(first(f1), first(f2)) + pair(second(f1), second(f2));
}

__device__ __forceinline__ void df_speeds(df u, df a, df &l1, df &l2, df &l3)
{
    const df eps = df(0.01) * a;
    l1 = entropy_fix(fabs(u + a), eps);
    l2 = entropy_fix(fabs(u - a), eps);
    l3 = entropy_fix(fabs(u), eps);
}

// source/flux.d:224-303; out: components (0, 3) and (1, 2)
__device__ __forceinline__ void roe_flux_df(const df qL[4], const df qR[4], df nx, df ny, dfp &o03, dfp &o12, df &sMax)
{
    DfSides S;
    dfp f03, f12;
    df_sides(qL, qR, nx, ny, S, f03, f12);
    const df di = sqrt(qR[0] * first(S.r));
    const df d1 = df(1.0f) / (df(1.0f) + di);
    const dfp n = pair(nx, ny);
    const dfp vel = (both(di) * pair(second(S.u), second(S.v)) + pair(first(S.u), first(S.v))) * both(d1);
    const df u = sum(vel * n);
    const df h = (di * second(S.h) + first(S.h)) * d1;
    const df vv = sum(vel * vel);
    df a, qq;
    split(root(pair(K<df>::gm1d * (h - half(vv)), vv)), a, qq);
    const dfp dm = pair(second(S.rv0), second(S.rv1)) - pair(first(S.rv0), first(S.rv1));
    const dfp dre = pair(qR[0], qR[3]) - pair(qL[0], qL[3]);
    df l1, l2, l3;
    df_speeds(u, a, l1, l2, l3);
    sMax = max4(fabs(l1), fabs(l2), fabs(l3), fabs(l3));
    const df s1 = half(l1 + l2), s2 = half(l1 - l2), sl = s1 - l3;
    df dRho, dRhoE;
    split(dre, dRho, dRhoE);
    const dfp t = pair(half(qq * qq), -u) * both(dRho) + pair(-sum(vel * dm), sum(dm * n));
    const df G1 = K<df>::gm1 * (first(t) + dRhoE), G2 = second(t);
    df ra, G1a2;  // 1 / a and G1 / a^2
    split(pair(df(1.0f), G1) / pair(a, a * a), ra, G1a2);
    const df C1 = sum(pair(G1a2, G2 * ra) * pair(sl, s2));
    const df C2 = sum(pair(G1 * ra, G2) * pair(s2, sl));
    const dfp l = both(l3), c = both(C1);
    dfp D03 = l * dre + pair(C1, C1 * h);
    const dfp D12 = l * dm + c * vel + both(C2) * n;
    D03 = pair(first(D03), second(D03) + C2 * u);
    o03 = half(f03) - half(D03);
    o12 = half(f12) - half(D12);
}

// source/flux.d:66-141, the reduced form of rusanov_flux
__device__ __forceinline__ void rusanov_flux_df(const df qL[4], const df qR[4], df nx, df ny, dfp &o03, dfp &o12, df &sMax)
{
    DfSides S;
    dfp f03, f12;
    df_sides(qL, qR, nx, ny, S, f03, f12);
    const df rho = sqrt(qL[0] * qR[0]);
    const dfp s = root(S.rho);
    const df rs = df(1.0f) / sum(s);
    const df vel0 = sum(s * S.u) * rs, vel1 = sum(s * S.v) * rs, p = sum(s * S.p) * rs;
    const df u = vel0 * nx + vel1 * ny;
    const df a = sqrt(K<df>::g * (p / rho));
    df l1, l2, l3;
    df_speeds(u, a, l1, l2, l3);
    const df sm = max4(fabs(l1), fabs(l2), fabs(l3), fabs(l3));
    sMax = sm;
    const dfp b = both(sm);
    const dfp dm = pair(second(S.rv0), second(S.rv1)) - pair(first(S.rv0), first(S.rv1));
    const dfp dre = pair(qR[0], qR[3]) - pair(qL[0], qL[3]);
    o03 = half(f03) - half(b * dre);
    o12 = half(f12) - half(b * dm);
}

// source/flux.d:28-64: components 3 and (1, 2) of the viscous flux; g[k]: the gradient of
// component k in (x, y).  The direction pair of a matrix row exchanges u and v (and the two
// coefficients of a pair) in its second element.
__device__ __forceinline__ void diffusive_flux_df(const ViscConst<df> &vc, df mu, const df q[4], const dfp g[4], df nx, df ny,
                                                  df &o3, dfp &o12)
{
    const df r = df(1.0f) / q[0];
    const dfp w = pair(q[1], q[2]) * both(r);  // (u, v)
    const dfp es = pair(q[3], mu) * both(r);   // E, mu / rho
    const df s = second(es);
    const dfp s2 = both(s), ww = w * w, uu = both(first(ww)), vv = both(second(ww)), u = both(first(w)), v = both(second(w));
    const dfp cross = swapped(w);
    const df c43 = df(-4.0 / 3.0), p43 = df(4.0 / 3.0), p23 = df(2.0 / 3.0), m23 = df(-2.0 / 3.0), c231 = df(2.0 / 3.0 - 1.0);
    const df gE = vc.gP * first(es);
    const dfp t = pair(vc.c43gP, vc.m1gP) * uu + pair(vc.m1gP, vc.c43gP) * vv - both(gE);
    const dfp z0 = g[0], z1 = g[1], z2 = g[2], z3 = g[3];
    const dfp w0 = swapped(z0), w1 = swapped(z1), w2 = swapped(z2);
    df x1, y1, x2, y2;
    split(z1, x1, y1);
    split(z2, x2, y2);
    // normal stresses of x in x and of y in y
    const dfp N = ((s2 * (both(c43) * w)) * z0 + both(s * p43) * pair(x1, y2)) +
                  ((s2 * (both(p23) * cross)) * w0 + both(s * m23) * pair(y2, x2));
    // work and heat in x and in y
    const df b30 = s * (c231 * first(w) * second(w));
    const dfp H = ((s2 * t) * z0 + (s2 * (pair(vc.p43mgP, vc.omgP) * u)) * z1 + (s2 * (pair(vc.omgP, vc.p43mgP) * v)) * z2 +
                   both(s * vc.gP) * z3) +
                  (both(b30) * w0 + (s2 * (pair(df(1.0f), m23) * v)) * w1 + (s2 * (pair(m23, df(1.0f)) * u)) * w2);
    // shear stress
    const dfp ns = both(-s);
    const df G = sum((ns * cross) * z0 + s2 * pair(x2, y1));
    const dfp n = pair(nx, ny);
    o12 = N * n + both(G) * swapped(n);
    o3 = sum(H * n);
}

}  // namespace ebbdev
