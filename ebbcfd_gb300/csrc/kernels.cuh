// kernels.cuh -- the explicit unstructured FV update as three kernels per stage,
// templated on the arithmetic type T:
//   T = double  plain FP64 path (k_fp64.cu, compiled without multiply-add contraction:
//               the reference's operation order, bitwise its results);
//   T = float   split path (k_split.cu): FP32 face, flux, gradient and limiter
//               arithmetic on FP32 copies of the FP64 geometry; the solution, the
//               u += dt R updates and the norm/force reductions stay FP64.
//   T = df      double-float path (k_df.cu): the same arithmetic on pairs of FP32
//               numbers (dfloat.h, ~46 bits) on double-float copies of the geometry,
//               stage states in double-float; the solution's update in the last
//               stage and the norm/force reductions stay FP64.
//
//   k_cell    one thread per interior cell: ghost states of its boundary faces
//             (solve.d:521-689), least-squares gradient and neighbour min/max
//             (solve.d:329-358), scalar and LP limiters (solve.d:360-497), and the
//             reconstructed state of each of its faces with the negative-pressure
//             fallback (solve.d:283-319,980-1011), written to that face's slot.
//   k_flux    one thread per edge: interior Roe/Rusanov (+viscous) flux from the two
//             face slots (solve.d:970-1033), boundary fluxes per BC (solve.d:769-968);
//             stores len*F and len*sMax once per edge.
//   k_update  one thread per interior cell: gathers its edges' len*F with the
//             +-1 multipliers in the cell's own edge order (the reference's summation
//             order), CFL time step, Rmax, -1/area scaling (solve.d:1080-1121), the
//             manufactured source, and the integrator stage combination
//             (integrators.d), with min/max/sum reductions in fixed-order trees;
//             split path: the freestream correction (uniform flow stays uniform).
// Accumulation is atomic-free (gather, not scatter); the only atomics are the
// order-independent min/max of dt and Rmax and the first-error key.  All three and
// the step epilogue use programmatic dependent launch (grid_dep_wait below).
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "bitconv.h"
#include "device_math.cuh"
#include "flux_df.cuh"
#include "flux_soft.cuh"
#include "layout.h"

namespace ebbdev {

constexpr int BC_FULLSTATE = 0, BC_CONSTP = 1, BC_INVWALL = 2, BC_VISCWALL = 3, BC_SYMMETRY = 4, BC_TPINFLOW = 5,
              BC_DIRICHLET = 6;
constexpr int BC_VERTICAL = 0x100;  // flag: reflection across a vertical edge (x1 == x2)
constexpr int ERR_NAN_EDGE = 8, ERR_NAN_CELL = 9, ERR_BC = 11;
// Threads per block and minimum resident blocks per SM requested through
// __launch_bounds__ (a register cap per thread: more warps in flight, possibly some
// spilling).  The FP32 (split) kernels are memory-latency bound and gain from it; the
// FP64 kernels are FP64-pipe bound.  Values and their timings in tuned.h, measured by
// ebbcfd_gb300/autotune.py (per-kernel event timing on GB300; 1 = the compiler's own
// register choice).
#include "tuned.h"
constexpr int UPD_THREADS = EBB_UPD_TB;
static_assert(EBB_UPD_TB == 256 || EBB_UPD_TB == 512, "k_update's block reductions take 256 or 512 threads");
// Launch shapes per arithmetic type and profile: _F split (float) on viscous meshes
// (tuned on the Navier-Stokes plate), _FI split on inviscid meshes (tuned on the Euler
// wedge: no stored gradients, fewer live values), _D plain FP64, _W double-float.  The
// profile PR (0 viscous or other forms, 1 split inviscid, 2 split inviscid on large meshes:
// shape_profile) is a template parameter of the stage kernels because the register cap is a
// compile-time launch bound.
#ifndef EBB_CELL_TB_FI
#define EBB_CELL_TB_FI 128
#endif
#ifndef EBB_CELL_MINB_FI
#define EBB_CELL_MINB_FI 8
#endif
#ifndef EBB_FLUX_TB_FI
#define EBB_FLUX_TB_FI 128
#endif
#ifndef EBB_FLUX_MINB_FI
#define EBB_FLUX_MINB_FI 12
#endif
#ifndef EBB_UPD_MINB_FI
#define EBB_UPD_MINB_FI 8
#endif
#ifndef EBB_FLUX_TB_W
#define EBB_FLUX_TB_W 128
#endif
#ifndef EBB_FLUX_MINB_W
#define EBB_FLUX_MINB_W 2
#endif
#ifndef EBB_UPD_MINB_W
#define EBB_UPD_MINB_W 3
#endif
// k_cell in FP64 and double-float takes first-order and LP-limited solves only (k_cell4 the
// others): the shapes it was tuned to on the plate while it took every solve
#define EBB_CELL_TB_D 128
#define EBB_CELL_MINB_D 6
#define EBB_CELL_TB_W 256
#define EBB_CELL_MINB_W 2
template <typename T, int PR> constexpr int pick(int f, int fi, int d, int w)
{
    return std::is_same<T, float>::value ? (PR ? fi : f) : (std::is_same<T, double>::value ? d : w);
}
template <typename T, int PR> constexpr int cell_threads()
{
    return pick<T, PR>(EBB_CELL_TB_F, EBB_CELL_TB_FI, EBB_CELL_TB_D, EBB_CELL_TB_W);
}
template <typename T, int PR> constexpr int flux_threads()
{
    return pick<T, PR>(EBB_FLUX_TB_F, EBB_FLUX_TB_FI, EBB_FLUX_TB_D, EBB_FLUX_TB_W);
}
template <typename T, int PR> constexpr int cell_minb()
{
    return pick<T, PR>(EBB_CELL_MINB_F, EBB_CELL_MINB_FI, EBB_CELL_MINB_D, EBB_CELL_MINB_W);
}
template <typename T, int PR> constexpr int flux_minb()
{
    return pick<T, PR>(EBB_FLUX_MINB_F, EBB_FLUX_MINB_FI, EBB_FLUX_MINB_D, EBB_FLUX_MINB_W);
}
template <typename T, int PR> constexpr int upd_minb()
{
    return pick<T, PR>(EBB_UPD_MINB_F, PR == 2 ? 8 : EBB_UPD_MINB_FI, EBB_UPD_MINB_D, EBB_UPD_MINB_W);
}
// k_cell4 (four threads per cell)
template <typename T> constexpr int cell4_threads() { return is_fp64<T> ? EBB_CELL4_TB_D : EBB_CELL4_TB_W; }
template <typename T> constexpr int cell4_minb() { return is_fp64<T> ? EBB_CELL4_MINB_D : EBB_CELL4_MINB_W; }
// an SM holds at most 2048 threads: every (threads, minimum blocks) pair must fit
static_assert(EBB_CELL_TB_F * EBB_CELL_MINB_F <= 2048 && EBB_CELL_TB_D * EBB_CELL_MINB_D <= 2048 &&
                  EBB_CELL_TB_FI * EBB_CELL_MINB_FI <= 2048,
              "k_cell bounds");
static_assert(EBB_CELL4_TB_D * EBB_CELL4_MINB_D <= 2048 && EBB_CELL4_TB_W * EBB_CELL4_MINB_W <= 2048 &&
                  EBB_CELL4_TB_D % 32 == 0 && EBB_CELL4_TB_W % 32 == 0,
              "k_cell4 bounds");
static_assert(EBB_FLUX_TB_F * EBB_FLUX_MINB_F <= 2048 && EBB_FLUX_TB_D * EBB_FLUX_MINB_D <= 2048 &&
                  EBB_FLUX_TB_FI * EBB_FLUX_MINB_FI <= 2048,
              "k_flux bounds");
static_assert(EBB_UPD_TB * EBB_UPD_MINB_F <= 2048 && EBB_UPD_TB * EBB_UPD_MINB_D <= 2048 &&
                  EBB_UPD_TB * EBB_UPD_MINB_FI <= 2048,
              "k_update bounds");
static_assert(EBB_CELL_TB_W * EBB_CELL_MINB_W <= 2048 && EBB_FLUX_TB_W * EBB_FLUX_MINB_W <= 2048 &&
                  EBB_UPD_TB * EBB_UPD_MINB_W <= 2048,
              "double-float bounds");


// Viscosity, Prandtl and CFL numbers in the arithmetic type: the split kernels read
// FP32 copies rounded once on the host or in the step epilogue (a per-thread FP64
// conversion occupies the FP64 pipe as long as an FP64 add)
template <typename T> __device__ __forceinline__ T visc_mu(const DMesh &M, const DPhys &P, int inst);
template <> __device__ __forceinline__ double visc_mu<double>(const DMesh &M, const DPhys &P, int inst)
{
    return M.inst_mu ? M.inst_mu[inst] : P.mu;
}
template <> __device__ __forceinline__ float visc_mu<float>(const DMesh &M, const DPhys &P, int inst)
{
    return M.inst_muf ? M.inst_muf[inst] : P.muf;
}
template <> __device__ __forceinline__ df visc_mu<df>(const DMesh &M, const DPhys &P, int inst)
{
    return M.inst_mu ? df(M.inst_mu[inst]) : P.muw;
}
template <typename T> __device__ __forceinline__ ViscConst<T> visc_const(const DPhys &P);
template <> __device__ __forceinline__ ViscConst<double> visc_const<double>(const DPhys &P)
{
    return {P.gP, P.c43gP, P.m1gP, P.p43mgP, P.omgP};
}
template <> __device__ __forceinline__ ViscConst<float> visc_const<float>(const DPhys &P)
{
    return visc_const_of<float>(P.prf);
}
template <> __device__ __forceinline__ ViscConst<df> visc_const<df>(const DPhys &P)
{
    return {P.gPw, P.c43gPw, P.m1gPw, P.p43mgPw, P.omgPw};
}
template <typename T> __device__ __forceinline__ T cfl_of(const DState *st)
{
    if constexpr (is_fp32<T>)
        return st->cflf;
    else
        return T(st->cfl);
}

__device__ __forceinline__ bool halted(const DState *st) { return st->done || st->err_key != EBB_NOERR; }

__device__ __forceinline__ void flag_error(DState *st, unsigned phase, unsigned code, unsigned idx)
{
    unsigned long long key = ((unsigned long long)phase << 48) | ((unsigned long long)code << 40) | idx;
    atomicMin(&st->err_key, key);
}

// Programmatic dependent launch.  The stage kernels and the step epilogue are
// launched with programmatic stream serialisation: a kernel's blocks may start while
// the previous kernel's last blocks still run, load the read-only mesh arrays (slot
// indices, geometry), and then wait at grid_dep_wait() until the previous kernel has
// completed and its writes are visible.  Every thread passes the wait before its
// first access to data another kernel writes and before it exits, so completion of a
// kernel implies completion of all kernels before it.  grid_dep_release() lets the
// next kernel start launching once every block of this one has issued it; it orders
// nothing.  In a launch without the attribute the wait returns at once.
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_dep_release() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// This launch's block of index blockIdx.x out of n: the kernels of a stage run through the
// mesh in opposite directions (DMesh::rev; k_cell always forward), so each starts with what
// the one before it has left in the L2 cache.  With the read-once arrays marked to leave it
// first (`stream`), no stored edge cells, the split update reading normals by edge instead
// of a copy by slot and wave speeds written and read in the stages that use them only: split
// steps of 1M plate cells 450 -> 437 us, of 500,000 triangles 91 -> 87 us (k_flux then writes
// 0.1 MB of its 15 MB to memory), double-float ones of 200,000 triangles 166 -> 149 us.
__device__ __forceinline__ int ordered_block(const DMesh &M, int n)
{
    return M.rev ? n - 1 - (int)blockIdx.x : (int)blockIdx.x;
}
// the cell of face slot s = j Cs + cell, j < 8
__device__ __forceinline__ int slot_cell(const DMesh &M, int s)
{
    const int Cs = M.Cs;
    if (M.maxJ > 4 && s >= 4 * Cs) s -= 4 * Cs;
    if (s >= 2 * Cs) s -= 2 * Cs;
    return s >= Cs ? s - Cs : s;
}

template <typename... KP, typename... AP>
inline cudaError_t launch_dep(void (*kernel)(KP...), dim3 grid, dim3 block, cudaStream_t s, AP... args)
{
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = 0;
    c.stream = s;
    c.attrs = at;
    c.numAttrs = 1;
    return cudaLaunchKernelEx(&c, kernel, args...);
}

// FP32 <-> FP64 conversions on the integer pipe (bitconv.h), for the split path
__device__ __forceinline__ double f2d_int(float x)
{
    const uint64_t b = ebbbits::f2d_bits(__float_as_uint(x));
    return __hiloint2double((int)(uint32_t)(b >> 32), (int)(uint32_t)b);
}
__device__ __forceinline__ float d2f_int(double x)
{
    return __uint_as_float(ebbbits::d2f_bits((uint32_t)__double2hiint(x), (uint32_t)__double2loint(x)));
}

// The FP64 value of a stage-kernel value and back.  Double-float: the word conversions
// on the integer pipe (exact), so each direction costs one FP64 add or subtract instead
// of two or three FP64-pipe conversions and an add; below FP32's normal range the
// words flush to zero, and an infinite or NaN value keeps a zero low word.
template <typename T> __device__ __forceinline__ double to_f64(T x) { return (double)x; }
template <> __device__ __forceinline__ double to_f64<df>(df x) { return f2d_int(x.hi) + f2d_int(x.lo); }
template <typename T> __device__ __forceinline__ T from_f64(double x) { return (T)x; }
template <> __device__ __forceinline__ df from_f64<df>(double x)
{
    const float h = d2f_int(x);
    const float l = d2f_int(x - f2d_int(h));
    return df(h, isfinite(h) ? l : 0.0f);
}

// 4-vector loads/stores: two 16-byte accesses for double, one for float
__device__ __forceinline__ void ld4(const double *p, double v[4])
{
    const double2 *q = reinterpret_cast<const double2 *>(p);
    double2 a = q[0], b = q[1];
    v[0] = a.x;
    v[1] = a.y;
    v[2] = b.x;
    v[3] = b.y;
}
__device__ __forceinline__ void st4(double *p, const double v[4])
{
    double2 *q = reinterpret_cast<double2 *>(p);
    q[0] = make_double2(v[0], v[1]);
    q[1] = make_double2(v[2], v[3]);
}
__device__ __forceinline__ void ld4(const float *p, float v[4])
{
    float4 a = *reinterpret_cast<const float4 *>(p);
    v[0] = a.x;
    v[1] = a.y;
    v[2] = a.z;
    v[3] = a.w;
}
__device__ __forceinline__ void st4(float *p, const float v[4])
{
    *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
// double-floats: (hi, lo) pairs, two 16-byte accesses per 4-vector as for double
__device__ __forceinline__ void ld4(const df *p, df v[4])
{
    const float4 *q = reinterpret_cast<const float4 *>(p);
    const float4 a = q[0], b = q[1];
    v[0] = df(a.x, a.y);
    v[1] = df(a.z, a.w);
    v[2] = df(b.x, b.y);
    v[3] = df(b.z, b.w);
}
__device__ __forceinline__ void st4(df *p, const df v[4])
{
    float4 *q = reinterpret_cast<float4 *>(p);
    q[0] = make_float4(v[0].hi, v[0].lo, v[1].hi, v[1].lo);
    q[1] = make_float4(v[2].hi, v[2].lo, v[3].hi, v[3].lo);
}
struct __align__(16) df2 {
    df x, y;
};
template <typename T> struct V2;
template <> struct V2<df> {
    using t = df2;
};
template <> struct V2<double> {
    using t = double2;
};
template <> struct V2<float> {
    using t = float2;
};
template <typename T> __device__ __forceinline__ typename V2<T>::t ld2(const void *base, size_t i)
{
    return reinterpret_cast<const typename V2<T>::t *>(base)[i];
}
template <typename T> __device__ __forceinline__ T ld1(const void *base, size_t i)
{
    return reinterpret_cast<const T *>(base)[i];
}
// the same for data a launch reads once and no other kernel of the stage reads: marked to
// leave the L2 cache first, so that what the next kernel reads stays
__device__ __forceinline__ float2 stream(const float2 *p) { return __ldcs(p); }
__device__ __forceinline__ double2 stream(const double2 *p) { return __ldcs(p); }
__device__ __forceinline__ int2 stream(const int2 *p) { return __ldcs(p); }
__device__ __forceinline__ int stream(const int *p) { return __ldcs(p); }
__device__ __forceinline__ df2 stream(const df2 *p)
{
    const float4 v = __ldcs(reinterpret_cast<const float4 *>(p));
    return {df(v.x, v.y), df(v.z, v.w)};
}
template <typename T> __device__ __forceinline__ typename V2<T>::t lds2(const void *base, size_t i)
{
    return stream(reinterpret_cast<const typename V2<T>::t *>(base) + i);
}
template <typename T> __device__ __forceinline__ const T *ptr(const void *base) { return reinterpret_cast<const T *>(base); }

// a / b and sqrt(x), FP64 on the integer pipe where the values allow it
template <typename T> __device__ __forceinline__ T ratio(T a, T b) { return a / b; }
template <> __device__ __forceinline__ double ratio<double>(double a, double b)
{
    return ebbdiv::div(a, ebbdiv::recip(b));
}
template <typename T> __device__ __forceinline__ T root(T x) { return dsqrt(x); }
template <> __device__ __forceinline__ double root<double>(double x)
{
    bool bad = false;
    const double r = ebbsoft::root(x, bad);
    return bad ? sqrt(x) : r;
}

template <typename T>
__device__ __forceinline__ void reflect(int type, const T *refl, T v0, T v1, T &o0, T &o1)
{
    if (type & BC_VERTICAL) {
        o0 = -v0;
        o1 = v1;
    } else {
        o0 = refl[0] * v0 + refl[1] * v1;
        o1 = refl[2] * v0 + refl[3] * v1;
    }
}

// ghost state of boundary edge b from the owner's state qi (solve.d:521-689)
template <typename T>
__device__ void ghost_state(const DMesh &M, const DPhys &P, DState *st, int b, const T qi[4], T qn[4])
{
    const int type = M.b_type[b];
    const T G = K<T>::g;
    switch (type & 0xff) {
    case BC_DIRICHLET:
        ld4(ptr<T>(M.g.b_dq) + 4 * (size_t)b, qn);
        break;
    case BC_FULLSTATE:
        for (int k = 0; k < 4; k++) qn[k] = qi[k];
        break;
    case BC_INVWALL:
    case BC_SYMMETRY: {
        T v0 = ratio(qi[1], qi[0]), v1 = ratio(qi[2], qi[0]), n0, n1;
        reflect(type, ptr<T>(M.g.b_refl) + 4 * (size_t)b, v0, v1, n0, n1);
        qn[0] = qi[0];
        qn[1] = qi[0] * n0;
        qn[2] = qi[0] * n1;
        qn[3] = qi[3];
        break;
    }
    case BC_VISCWALL:
        qn[0] = qi[0];
        qn[1] = -qi[1];
        qn[2] = -qi[2];
        qn[3] = qi[3];
        break;
    case BC_CONSTP: {
        T rhop = qi[0], up = ratio(qi[1], qi[0]), vp = ratio(qi[2], qi[0]);
        T pp = pressure(qi);
        T ap = root(G * ratio(pp, rhop));
        T Jp = up + ratio(T(2.0) * ap, G - 1);
        T Sp = ratio(pp, dpow(rhop, G));
        T pb = ptr<T>(M.g.b_data)[4 * (size_t)b];
        T rhob = dpow(ratio(pb, Sp), T(1.0 / 1.4));
        T ab = root(G * ratio(pb, rhob));
        T ub = Jp - ratio(T(2.0) * ab, G - 1);
        T vb = vp;
        T mag = root(ub * ub + vb * vb);
        T rEb = ratio(pb, G - 1) + T(0.5) * rhob * (mag * mag);
        const typename V2<T>::t n = ld2<T>(M.g.b_n, b);
        T vpn = up * n.x + vp * n.y;
        T vbn = ub * n.x + vb * n.y;
        T g0 = up - vpn * n.x + vbn * n.x;
        T g1 = vp - vpn * n.y + vbn * n.y;
        qn[0] = rhob;
        qn[1] = rhob * g0;
        qn[2] = rhob * g1;
        qn[3] = rEb;
        break;
    }
    case BC_TPINFLOW: {
        const T *bd = ptr<T>(M.g.b_data) + 4 * (size_t)b;
        T Tt = bd[0], Pt = bd[1], nin0 = bd[2], nin1 = bd[3];
        T rhop = qi[0], up = qi[1] / qi[0];
        T pp = pressure(qi);
        T ap = dsqrt(G * (pp / rhop));
        T Jp = up + (T(2.0) * ap) / (G - 1);
        const typename V2<T>::t n = ld2<T>(M.g.b_n, b);
        T d = nin0 * n.x + nin1 * n.y;
        T Rg = (T)P.r_gas;
        T aa = G * Rg * Tt * (d * d) - T(0.5) * (G - 1) * (Jp * Jp);
        T bb = (T(4.0) * G * Rg * Tt * d) / (G - 1);
        T cc = (T(4.0) * G * Rg * Tt) / ((G - 1) * (G - 1)) - Jp * Jp;
        T M1 = (-bb + dsqrt(bb * bb - 4 * aa * cc)) / (T(2.0) * aa);
        T M2 = (-bb - dsqrt(bb * bb - 4 * aa * cc)) / (T(2.0) * aa);
        T Mb = 0;
        if (M1 >= 0 && M2 >= 0)
            Mb = fmin(M1, M2);
        else if (M1 >= 0 && M2 < 0)
            Mb = M1;
        else if (M1 < 0 && M2 >= 0)
            Mb = M2;
        else
            flag_error(st, 0, ERR_BC, (unsigned)M.b_ref[b]);
        T Tb = Tt / (1 + T(0.5) * (G - 1) * (Mb * Mb));
        T pb = Pt * dpow(Tb / Tt, G / (G - 1));
        T rhob = pb / (Rg * Tb);
        T ab = dsqrt(G * (pb / rhob));
        T vb0 = Mb * ab * nin0, vb1 = Mb * ab * nin1;
        T mag = dsqrt(vb0 * vb0 + vb1 * vb1);
        T rEb = pb / (G - 1) + T(0.5) * rhob * (mag * mag);
        // solve.d:678-681 writes every value into component 0; the other
        // components of the ghost slot are never written and stay zero
        qn[0] = rEb;
        qn[1] = 0;
        qn[2] = 0;
        qn[3] = 0;
        break;
    }
    default:
        for (int k = 0; k < 4; k++) qn[k] = qi[k];
    }
}

// LP!m (solve.d:37-173) on the m = 4 + 2*nNb constraints of solve.d:404-497
template <typename T>
__device__ __forceinline__ void lp_limit(const DMesh &M, int i, int ne, const T qi[4], const T mn[4], const T mx[4],
                                         const T g[4][2], T lim0[4], T lim1[4], T thresh)
{
#pragma unroll 1
    for (int k = 0; k < 4; k++) {
        if (!(lim0[k] < thresh) || !(ne == 3 || ne == 4)) continue;
        T A[12][2], b[12];
        int mr = 4 + 2 * ne;
        A[0][0] = 1;
        A[0][1] = 0;
        A[1][0] = 0;
        A[1][1] = 1;
        A[2][0] = -1;
        A[2][1] = 0;
        A[3][0] = 0;
        A[3][1] = -1;
        b[0] = 0;
        b[1] = 0;
        b[2] = -1;
        b[3] = -1;
        for (int j = 0; j < ne; j++) {
            const typename V2<T>::t nd = ld2<T>(M.g.s_nd, (size_t)j * M.Cs + i);
            A[2 * j + 4][0] = nd.x * g[k][0];
            A[2 * j + 4][1] = nd.y * g[k][1];
            b[2 * j + 4] = mn[k] - qi[k];
            A[2 * j + 5][0] = -nd.x * g[k][0];
            A[2 * j + 5][1] = -nd.y * g[k][1];
            b[2 * j + 5] = qi[k] - mx[k];
        }
        T c0 = -fabs(g[k][0]), c1 = -fabs(g[k][1]);
        T xk0 = 0, xk1 = 0;
        int W0 = 0, W1 = 1;
        T Ak[4] = {A[0][0], A[0][1], A[1][0], A[1][1]};
        for (int it = 0;;) {
            T det = Ak[0] * Ak[3] - Ak[1] * Ak[2];
            T id = T(1.0) / det;
            T l0 = (Ak[3] * id) * c0 + (-Ak[2] * id) * c1;
            T l1 = (-Ak[1] * id) * c0 + (Ak[0] * id) * c1;
            if ((l0 >= T(-10e-9)) && (l1 >= T(-10e-9))) break;
            int qi_ = (l0 < l1) ? W0 : W1;
            T e0 = (l0 < l1) ? 1 : 0, e1 = (l0 < l1) ? 0 : 1;
            T pk0 = (Ak[3] * id) * e0 + (-Ak[1] * id) * e1;
            T pk1 = (-Ak[2] * id) * e0 + (Ak[0] * id) * e1;
            T alpha = INFINITY;
            int t = 0;
            T gam[12];
            int D[12], Dlen = 0;
            for (int r = 0; r < mr; r++)
                if (r != W0 && r != W1)
                    if (A[r][0] * pk0 + A[r][1] * pk1 < T(-1e-11)) D[Dlen++] = r;
            for (int r = 0; r < Dlen; r++) {
                T aixk = A[D[r]][0] * xk0 + A[D[r]][1] * xk1;
                T aipk = A[D[r]][0] * pk0 + A[D[r]][1] * pk1;
                gam[r] = (aixk - b[D[r]]) / (-aipk);
                alpha = fmin(alpha, gam[r]);
            }
            for (int r = 0; r < Dlen; r++)
                if (gam[r] == alpha) {
                    t = D[r];
                    break;
                }
            if (qi_ == W0)
                W0 = t;
            else if (qi_ == W1)
                W1 = t;
            Ak[0] = A[W0][0];
            Ak[1] = A[W0][1];
            Ak[2] = A[W1][0];
            Ak[3] = A[W1][1];
            xk0 += alpha * pk0;
            xk1 += alpha * pk1;
            if (++it > 15) break;
        }
        lim0[k] = xk0;
        lim1[k] = xk1;
    }
}

// read-only mesh data of a cell loaded before the wait for the previous kernel (split
// path): neighbour indices, gradient weights, neighbour and face midpoint offsets
template <typename T, int MJ> struct CellPre {
    int nb[MJ];
    typename V2<T>::t gm[MJ], nd[MJ], fd[MJ];
};

template <typename T, int MJ, bool LP>
__device__ __forceinline__ void cell_body(const DMesh &M, const DPhys &P, const DArrays &A, DState *st, int i, int ne,
                                          const T *__restrict__ qin, int limit, CellPre<T, MJ> &pre)
{
    const int Cs = M.Cs;
    T *qghost = const_cast<T *>(qin);  // ghost slots [C, C+G) are written by their owner only
    T qi[4];
    ld4(qin + 4 * (size_t)i, qi);
    T mn[4], mx[4], g[4][2];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        mn[k] = qi[k];
        mx[k] = qi[k];
        g[k][0] = T(0.0);
        g[k][1] = T(0.0);
    }
    const bool second = P.order > 1;
    if constexpr (sizeof(T) == 4) {
        // all neighbour-state gathers in flight before any dependent math
        T qv[MJ][4];
#pragma unroll
        for (int j = 0; j < MJ; j++) pre.nb[j] = (j < ne) ? pre.nb[j] : i;
#pragma unroll
        for (int j = 0; j < MJ; j++) ld4(qin + 4 * (size_t)(pre.nb[j] < M.C ? pre.nb[j] : i), qv[j]);
#pragma unroll
        for (int j = 0; j < MJ; j++) {
            if (j < ne) {
                if (pre.nb[j] >= M.C) {
                    ghost_state<T>(M, P, st, pre.nb[j] - M.C, qi, qv[j]);
                    st4(qghost + 4 * (size_t)pre.nb[j], qv[j]);
                }
                if (second) {
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        mn[k] = fmin(mn[k], qv[j][k]);
                        mx[k] = fmax(mx[k], qv[j][k]);
                        T du = qv[j][k] - qi[k];
                        g[k][0] = g[k][0] + pre.gm[j].x * du;
                        g[k][1] = g[k][1] + pre.gm[j].y * du;
                    }
                }
            }
        }
    } else if constexpr (is_df<T>) {
        // double-float: the neighbour-state gathers in flight before the arithmetic,
        // which keeps the FP64 path's order (long dependent FP32 sequences leave the
        // warps waiting on one gather at a time otherwise)
        int nb[MJ];
        T qv[MJ][4];
#pragma unroll
        for (int j = 0; j < MJ; j++) nb[j] = (j < ne) ? M.s_nbr[(size_t)j * Cs + i] : i;
#pragma unroll
        for (int j = 0; j < MJ; j++) ld4(qin + 4 * (size_t)(nb[j] < M.C ? nb[j] : i), qv[j]);
#pragma unroll
        for (int j = 0; j < MJ; j++) {
            if (j < ne) {
                if (nb[j] >= M.C) {
                    ghost_state<T>(M, P, st, nb[j] - M.C, qi, qv[j]);
                    st4(qghost + 4 * (size_t)nb[j], qv[j]);
                }
                if (second) {
                    const typename V2<T>::t gm = ld2<T>(M.g.s_gm, (size_t)j * Cs + i);
#pragma unroll
                    for (int k = 0; k < 4; k++) {
                        mn[k] = fmin(mn[k], qv[j][k]);
                        mx[k] = fmax(mx[k], qv[j][k]);
                        T du = qv[j][k] - qi[k];
                        g[k][0] = g[k][0] + gm.x * du;
                        g[k][1] = g[k][1] + gm.y * du;
                    }
                }
            }
        }
    } else {
#pragma unroll
    for (int j = 0; j < MJ; j++) {
        if (j < ne) {
            const size_t s = (size_t)j * Cs + i;
            const int nb = M.s_nbr[s];
            T qn[4];
            if (nb < M.C) {
                ld4(qin + 4 * (size_t)nb, qn);
            } else {
                ghost_state<T>(M, P, st, nb - M.C, qi, qn);
                st4(qghost + 4 * (size_t)nb, qn);
            }
            if (second) {
                const typename V2<T>::t gm = ld2<T>(M.g.s_gm, s);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    mn[k] = fmin(mn[k], qn[k]);
                    mx[k] = fmax(mx[k], qn[k]);
                    T du = qn[k] - qi[k];
                    g[k][0] = g[k][0] + gm.x * du;
                    g[k][1] = g[k][1] + gm.y * du;
                }
            }
        }
    }
    }
    T lim0[4] = {T(1.0), T(1.0), T(1.0), T(1.0)}, lim1[4] = {T(1.0), T(1.0), T(1.0), T(1.0)};
    if (second && P.limited && limit && sizeof(T) == 8) {
        // FP64: the out-of-bounds tests first, then only the needed divisions in a
        // compact loop.  Branching on each (neighbour, component) pair makes a warp run
        // a division whenever any of its lanes needs it, and an FP64 division costs
        // about ten FP64-unit instructions per warp; the compact loop runs as many as
        // the busiest lane needs.  Each component's limiter still takes the minimum in
        // neighbour order (pairs in bounds give s = 1, which leaves it unchanged).
        unsigned need = 0, above = 0;
        // FP64: each test is first taken in FP32 from the values truncated on the
        // integer pipe (trunc_sat: within 2^-23, tiny values to zero, huge ones to
        // infinity).  The FP32 qE is within 2^-20 of S = |q| + |g0 nx| + |g1 ny| of the
        // FP64 one, so a side clear of 2^-18 S + 2^-100 (and 2^-20 of each bound) is
        // the FP64 expression's; pairs closer to a bound (in uniform regions every
        // pair), and NaN or overflowing ones, take the FP64 expression.
        float qf[4], g0f[4], g1f[4], lof[4], hif[4];
        if constexpr (is_fp64<T>) {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                qf[k] = trunc_sat(qi[k]);
                g0f[k] = trunc_sat(g[k][0]);
                g1f[k] = trunc_sat(g[k][1]);
                lof[k] = trunc_sat(mn[k]);
                hif[k] = trunc_sat(mx[k]);
            }
        }
#pragma unroll
        for (int j = 0; j < MJ; j++) {
            if (j < ne) {
                const typename V2<T>::t nd = ld2<T>(M.g.s_nd, (size_t)j * Cs + i);
                float nxf = 0.0f, nyf = 0.0f;
                if constexpr (is_fp64<T>) {
                    nxf = trunc_sat(nd.x);
                    nyf = trunc_sat(nd.y);
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const unsigned bit = 1u << (4 * j + k);
                    int side = -1;
                    if constexpr (is_fp64<T>) {
                        const float a = __fmul_rn(g0f[k], nxf), b = __fmul_rn(g1f[k], nyf);
                        const float e = __fadd_rn(qf[k], __fadd_rn(a, b));
                        const float B = __fadd_rn(0x1p-18f * __fadd_rn(__fadd_rn(fabsf(qf[k]), fabsf(a)), fabsf(b)), 0x1p-100f);
                        const float bl = __fadd_rn(0x1p-20f * fabsf(lof[k]), 0x1p-100f);
                        const float bh = __fadd_rn(0x1p-20f * fabsf(hif[k]), 0x1p-100f);
                        if (__fsub_rn(e, B) > __fadd_rn(lof[k], bl) && __fadd_rn(e, B) < __fsub_rn(hif[k], bh))
                            side = 0;
                        else if (__fadd_rn(e, B) < __fsub_rn(lof[k], bl))
                            side = 1;
                        else if (__fsub_rn(e, B) > __fadd_rn(hif[k], bh))
                            side = 2;
                    }
                    if (side < 0) {
                        const T qE = qi[k] + (g[k][0] * nd.x + g[k][1] * nd.y);
                        side = qE < mn[k] ? 1 : (qE > mx[k] ? 2 : 0);
                    }
                    if (side) need |= bit;
                    if (side == 2) above |= bit;
                }
            }
        }
        while (need) {
            const int t = __ffs(need) - 1;
            const unsigned bit = 1u << t;
            need &= need - 1;
            const int j = t >> 2, k = t & 3;
            const typename V2<T>::t nd = ld2<T>(M.g.s_nd, (size_t)j * Cs + i);
            T g0 = g[0][0], g1 = g[0][1], q = qi[0], lo = mn[0], hi = mx[0], l = lim0[0];
#pragma unroll
            for (int kk = 1; kk < 4; kk++)
                if (k == kk) {
                    g0 = g[kk][0];
                    g1 = g[kk][1];
                    q = qi[kk];
                    lo = mn[kk];
                    hi = mx[kk];
                    l = lim0[kk];
                }
            const T s = ((above & bit) ? hi - q : lo - q) / (g0 * nd.x + g1 * nd.y);
            l = fmin(l, s);
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
                if (k == kk) lim0[kk] = l;
        }
#pragma unroll
        for (int k = 0; k < 4; k++) lim1[k] = lim0[k];
        if (LP) lp_limit<T>(M, i, ne, qi, mn, mx, g, lim0, lim1, (T)P.lp_thresh);
    } else if (second && P.limited && limit) {
#pragma unroll
        for (int j = 0; j < MJ; j++) {
            if (j < ne) {
                typename V2<T>::t nd;
                if constexpr (sizeof(T) == 4)
                    nd = pre.nd[j];
                else
                    nd = ld2<T>(M.g.s_nd, (size_t)j * Cs + i);
                // every pair's quotient is formed and selected (no divergent branch; the
                // FP32 division is a reciprocal and a multiply): pairs in bounds leave the
                // limiter unchanged, as s = 1 does in solve.d:360-402
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const T dd = g[k][0] * nd.x + g[k][1] * nd.y;
                    const T qE = qi[k] + dd;
                    const bool lo = qE < mn[k], hi = qE > mx[k];
                    const T s = ((lo ? mn[k] : mx[k]) - qi[k]) / dd;
                    lim0[k] = (lo || hi) ? fmin(lim0[k], s) : lim0[k];
                    lim1[k] = lim0[k];
                }
            }
        }
        if (LP) lp_limit<T>(M, i, ne, qi, mn, mx, g, lim0, lim1, (T)P.lp_thresh);
    }
    if (P.need_grad) {
        T *gp = reinterpret_cast<T *>(A.grad) + 8 * (size_t)i;
        if (second) {
            T a[4] = {g[0][0], g[0][1], g[1][0], g[1][1]}, b[4] = {g[2][0], g[2][1], g[3][0], g[3][1]};
            st4(gp, a);
            st4(gp + 4, b);
        } else {  // order 1: interior gradients are never computed (NaN-initialised in the reference)
            T nanv[4] = {T(NAN), T(NAN), T(NAN), T(NAN)};
            st4(gp, nanv);
            st4(gp + 4, nanv);
        }
    }
    if (A.lim) {  // limiter values, exported for ebb-reconstruct
        T *lp = reinterpret_cast<T *>(A.lim) + 8 * (size_t)i;
        T a[4] = {lim0[0], lim1[0], lim0[1], lim1[1]}, b[4] = {lim0[2], lim1[2], lim0[3], lim1[3]};
        st4(lp, a);
        st4(lp + 4, b);
    }
    T lg0[4], lg1[4];
    T l0 = T(1.0), l1 = T(1.0);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        lg0[k] = lim0[k] * g[k][0];
        lg1[k] = lim1[k] * g[k][1];
        l0 = fmin(l0, lim0[k]);
        l1 = fmin(l1, lim1[k]);
    }
    T *face = reinterpret_cast<T *>(A.face);
#pragma unroll
    for (int j = 0; j < MJ; j++) {
        if (j < ne) {
            const size_t s = (size_t)j * Cs + i;
            T f[4];
            if (!second) {
#pragma unroll
                for (int k = 0; k < 4; k++) f[k] = qi[k];
            } else {
                typename V2<T>::t fd;
                if constexpr (sizeof(T) == 4)
                    fd = pre.fd[j];
                else
                    fd = ld2<T>(M.g.s_fd, s);
#pragma unroll
                for (int k = 0; k < 4; k++) f[k] = qi[k] + lg0[k] * fd.x + lg1[k] * fd.y;
                if (pressure_negative(f)) {
                    const int ev = M.s_edge[s] & 0x7fffffff;
                    const T ll1 = (ev >= M.Eint) ? l0 : l1;  // updateBoundaryEdge uses lim[0] twice
#pragma unroll
                    for (int k = 0; k < 4; k++) f[k] = qi[k] + l0 * g[k][0] * fd.x + ll1 * g[k][1] * fd.y;
                }
            }
            st4(face + 4 * s, f);
        }
    }
}

// plain FP64: the cells k_cell4 leaves
template <typename T, int MJ, bool LP>
__device__ __noinline__ void cell_plain(const DMesh &M, const DPhys &P, const DArrays &A, DState *st, int i, int ne,
                                        const T *qin, int limit)
{
    CellPre<T, MJ> pre;
    cell_body<T, MJ, LP>(M, P, A, st, i, ne, qin, limit, pre);
}

// The scalar limiter of one component (solve.d:336-402) on the integer and FP32 pipes.
// lo <= 0 <= hi are FP32 values of the bounds minus the cell's value (lo0, hi0: exactly
// zero), g0f and g1f of the gradient (flat: exactly zero).  Which neighbours' extrapolations
// leave the bounds, and which of those gives the smallest ratio, is decided in FP32 from
// values good to 23 bits; a decision that is not clear of their errors and of M, the
// rounding of the cell's value plus a difference, sets `unsure` (limit_exact then decides;
// measured on smooth flows: 2 to 3 of 1,000 cells).  Returns the deciding neighbour, or -1;
// `low` tells its bound.
//
// With dd = g0 nx + g1 ny in the form's arithmetic and e its FP32 value: |e - dd| < 2^-21
// (|a| + |b|), the FP32 bounds are within 2^-23 of theirs, and q + dd compares with a bound
// as dd does with its difference when they are M / 2 apart (FP64: 2^-51 |q|).
template <int MJ>
__device__ __forceinline__ int limiting_neighbour(float M, float g0f, float g1f, bool flat, float lo, float hi, bool lo0,
                                                  bool hi0, const float (&nx)[MJ], const float (&ny)[MJ], int ne,
                                                  bool &low, bool &unsure)
{
    const float ml = __fmaf_rn(0x1p-21f, fabsf(lo), M), mh = __fmaf_rn(0x1p-21f, hi, M);
    const float lo_out = lo - ml, lo_in = lo + ml, hi_out = hi + mh, hi_in = hi - mh;
    int best = -1;
    float s1 = 4.0f, up1 = 4.0f, dn1 = 4.0f, dn2 = 8.0f;  // the smallest ratio and its interval, the others' lower end
#pragma unroll
    for (int j = 0; j < MJ; j++) {
        if (j < ne) {
            const float a = __fmul_rn(g0f, nx[j]), b = __fmul_rn(g1f, ny[j]), e = __fadd_rn(a, b);
            const float E = __fmul_rn(0x1p-20f, __fadd_rn(fabsf(a), fabsf(b)));
            const float up = e + E, dn = e - E;
            const bool below = up < lo_out, above = dn > hi_out, in = dn > lo_in && up < hi_in;
            unsure |= !((below || above || in) && fabsf(e) < 0x1p100f) && !flat;
            if (below || above) {
                const float r = __fdividef(1.0f, e), s = (below ? lo : hi) * r;
                const float w = s * __fmaf_rn(2.0f * E, fabsf(r), 0x1p-20f);
                if (s < s1) {
                    dn2 = fminf(dn2, dn1);
                    s1 = s;
                    up1 = s + w;
                    dn1 = s - w;
                    best = j;
                    low = below;
                } else {
                    dn2 = fminf(dn2, s - w);
                }
            }
        }
    }
    // two ratios too close to tell apart (a zero one is the smallest: its bound is exact)
    if (best >= 0) unsure |= !(low ? lo0 : hi0) && !(s1 > 0x1p-60f && dn2 > up1);
    return best;
}

// The limiter of component k in the reference's own expressions (solve.d:336-402), the
// neighbours' values read again (ghosts as this thread has just written them).
__device__ __forceinline__ double limit_exact(const DMesh &M, int i, int ne, const double *qin, int k, double q, double g0,
                                              double g1)
{
    double mn = q, mx = q, l = 1.0;
#pragma unroll 1
    for (int j = 0; j < ne; j++) {
        const double v = *(const volatile double *)(qin + 4 * (size_t)M.s_nbr[(size_t)j * M.Cs + i] + k);
        mn = fmin(mn, v);
        mx = fmax(mx, v);
    }
#pragma unroll 1
    for (int j = 0; j < ne; j++) {
        const double2 nd = ld2<double>(M.g.s_nd, (size_t)j * M.Cs + i);
        const double dd = g0 * nd.x + g1 * nd.y, qE = q + dd;
        if (qE < mn || qE > mx) l = fmin(l, ebbdiv::div((qE < mn ? mn : mx) - q, ebbdiv::recip(dd)));
    }
    return l;
}

__device__ __forceinline__ df limit_exact(const DMesh &M, int i, int ne, df g0, df g1, df dl, df dh)
{
    df l = df(1.0f);
#pragma unroll 1
    for (int j = 0; j < ne; j++) {
        const df2 nd = ld2<df>(M.g.s_nd, (size_t)j * M.Cs + i);
        const df dd = g0 * nd.x + g1 * nd.y;
        if (dd < dl || dd > dh) l = fmin(l, (dd < dl ? dl : dh) / dd);
    }
    return l;
}

// pressure_negative of a face state whose four components sit in the four lanes of a
// quad (x: this lane's, k its index), the same answer in each of them
__device__ __forceinline__ bool pressure_negative4(double x, int k, unsigned quad)
{
    const bool ok = (k == 0 || k == 3) ? mid_range(x, true) : f32_range(x);
    const float t = ok ? trunc_sat(x) : NAN;
    const float r = __shfl_sync(quad, t, 0, 4), m1 = __shfl_sync(quad, t, 1, 4), m2 = __shfl_sync(quad, t, 2, 4),
                e = __shfl_sync(quad, t, 3, 4);
    const float W = __fmul_rn(e, r), Z = __fmul_rn(0.5f, __fadd_rn(__fmul_rn(m1, m1), __fmul_rn(m2, m2)));
    const float d = __fsub_rn(W, Z);
    if (fabsf(d) > 0x1p-17f * __fadd_rn(fabsf(W), Z)) return d < 0.0f;
    const double q[4] = {__shfl_sync(quad, x, 0, 4), __shfl_sync(quad, x, 1, 4), __shfl_sync(quad, x, 2, 4),
                         __shfl_sync(quad, x, 3, 4)};
    return pressure_negative(q);
}
__device__ __forceinline__ df shfl4(unsigned quad, df x, int k)
{
    return df(__shfl_sync(quad, x.hi, k, 4), __shfl_sync(quad, x.lo, k, 4));
}
__device__ __forceinline__ double shfl4(unsigned quad, double x, int k) { return __shfl_sync(quad, x, k, 4); }
__device__ __forceinline__ bool pressure_negative4(df x, int, unsigned quad)
{
    const float r = __shfl_sync(quad, x.hi, 0, 4), m1 = __shfl_sync(quad, x.hi, 1, 4), m2 = __shfl_sync(quad, x.hi, 2, 4),
                e = __shfl_sync(quad, x.hi, 3, 4);
    const float W = e * r, Z = 0.5f * (m1 * m1 + m2 * m2), d = W - Z;
    if (r > 0.0f && fabsf(d) > 0x1p-17f * (fabsf(W) + Z) + 0x1p-100f) return d < 0.0f;
    const df q[4] = {shfl4(quad, x, 0), shfl4(quad, x, 1), shfl4(quad, x, 2), shfl4(quad, x, 3)};
    return pressure_negative(q);
}

// Gradient, scalar limiter and face states with four threads per cell, one per component
// (plain FP64 and double-float; second order, without the LP limiter).  The components
// meet only in the ghost states and the pressure test of a face, so a thread carries a
// quarter of the values: the registers of one thread per cell (80 and 128 of them) kept
// 24 and 16 warps on an SM, too few to cover the latency of either form's arithmetic.
//
// The limiter's decisions are taken in FP32 (limiting_neighbour), so that one quotient per
// component is formed.  FP64: the products and that quotient run on the integer pipe
// (softdbl.h) beside the FP64 pipe; the values are cell_body's bit for bit, and a cell with
// a value out of that arithmetic's range goes to cell_plain.  Bound by the FP64 pipe's
// additions and the integer pipe (56% and 56% busy on 1M plate cells, 50% and 61% on 1M
// triangles; a sixth of the time fetching instructions).
// Double-float: x and y in packed operations (dfpair.cuh), bound by issue.
//
// Lane k loads the geometry of slot k before the wait for the previous kernel: with each
// lane loading every slot's where it is used, loads from memory took 45% (FP64) and 63%
// (double-float) of the warps' time.
//
// Measured against one thread per cell, us per launch, FP64 / double-float: 400,000 plate
// cells 147 (318 all on the FP64 pipe, 143 as here) / 80 (109); 200,000 triangles 55 (155,
// 52) / 25 (36); 1024 quads, where one warp's latency is the launch's, 7.3 (23, 16) / 5.1
// (14).
template <typename T, int MJ, bool UNI>
__global__ void __launch_bounds__(cell4_threads<T>(), cell4_minb<T>())
    k_cell4(const __grid_constant__ DMesh M, const __grid_constant__ DPhys P, const __grid_constant__ DArrays A,
            const T *__restrict__ qin, int limit)
{
    const int t = ordered_block(M, gridDim.x) * blockDim.x + threadIdx.x;
    const int i = t >> 2, k = t & 3;
    const bool act = i < M.C;
    const int Cs = M.Cs;
    // read-only mesh data before the wait for the previous kernel: lane k holds the slots
    // k and k + 4 of its cell (rows past the cell's edges hold 0), so that every load is in
    // flight at once; the quad passes them around
    constexpr int H = MJ > 4 ? 2 : 1;
    int ne = 0, inst = 0, nbk[H] = {};
    typename V2<T>::t gmk[H] = {}, ndk[H] = {}, fdk[H] = {};
    if (act) {
        ne = UNI ? MJ : M.nedge[i];
        if (M.cell_inst) inst = M.cell_inst[i];
#pragma unroll
        for (int h = 0; h < H; h++) {
            if (4 * h + k < MJ) {
                const size_t s = (size_t)(4 * h + k) * Cs + i;
                nbk[h] = stream(M.s_nbr + s);
                gmk[h] = lds2<T>(M.g.s_gm, s);
                ndk[h] = lds2<T>(M.g.s_nd, s);
                fdk[h] = lds2<T>(M.g.s_fd, s);
            }
        }
    }
    grid_dep_release();
    grid_dep_wait();
    if (!act) return;  // a quad's lanes agree here and below
    DState *st = A.st + inst;
    const unsigned quad = 0xfu << (threadIdx.x & 28);
    T *qghost = const_cast<T *>(qin);  // ghost slots [C, C+G) are written by their owner only
    const T qi = qin[4 * (size_t)i + k];
    int nb[MJ];
    T qv[MJ];
#pragma unroll
    for (int j = 0; j < MJ; j++) {
        nb[j] = __shfl_sync(quad, nbk[j >> 2], j & 3, 4);
        if (UNI || j < ne) qv[j] = qin[4 * (size_t)(nb[j] < M.C ? nb[j] : i) + k];
    }
    if (halted(st)) return;  // behind the gathers: they and this test wait together
    auto slot = [&](const typename V2<T>::t(&v)[H], int j) {  // slot j's pair, j a constant
        typename V2<T>::t o;
        o.x = shfl4(quad, v[j >> 2].x, j & 3);
        o.y = shfl4(quad, v[j >> 2].y, j & 3);
        return o;
    };
    bool bad = false;
    T g0 = T(0.0), g1 = T(0.0), dl = T(0.0), dh = T(0.0);  // smallest and largest neighbour difference, or 0
    long long dlo = 0, dhi = 0;                            // FP64: their bit patterns
    dfp gp = pair(df(0.0f), df(0.0f));                     // double-float: the gradient
#pragma unroll
    for (int j = 0; j < MJ; j++) {
        if (UNI || j < ne) {
            if (nb[j] >= M.C) {
                const T q[4] = {shfl4(quad, qi, 0), shfl4(quad, qi, 1), shfl4(quad, qi, 2), shfl4(quad, qi, 3)};
                T gh[4];
                ghost_state<T>(M, P, st, nb[j] - M.C, q, gh);
                qv[j] = k < 2 ? (k ? gh[1] : gh[0]) : (k == 2 ? gh[2] : gh[3]);
                qghost[4 * (size_t)nb[j] + k] = qv[j];
            }
            const typename V2<T>::t gm = slot(gmk, j);
            const T du = qv[j] - qi;
            if constexpr (is_fp64<T>) {
                ebbsoft::check<200>(du, bad);
                // negative doubles are larger than others as unsigned integers, the more
                // the larger their magnitude; non-negative ones order as signed integers
                const long long bits = __double_as_longlong(du);
                dlo = (unsigned long long)bits > (unsigned long long)dlo ? bits : dlo;
                dhi = bits > dhi ? bits : dhi;
                const double px = ebbsoft::mul(gm.x, du), py = ebbsoft::mul(gm.y, du);
                g0 = j == 0 ? zero_plus(px) : g0 + px;
                g1 = j == 0 ? zero_plus(py) : g1 + py;
            } else {
                if (du < dl) dl = du;
                if (du > dh) dh = du;
                const dfp p = pair(gm.x, gm.y) * both(du);
                gp = j == 0 ? p : gp + p;
            }
        }
    }
    float g0f, g1f, lo, hi, mar;
    if constexpr (is_fp64<T>) {
        ebbsoft::check<200>(g0, bad);
        ebbsoft::check<200>(g1, bad);
        dl = dlo < 0 ? __longlong_as_double(dlo) : 0.0;
        dh = __longlong_as_double(dhi);
        g0f = trunc_sat(g0);
        g1f = trunc_sat(g1);
        lo = trunc_sat(dl);
        hi = trunc_sat(dh);
        mar = __fadd_rn(0x1p-50f * fabsf(trunc_sat(qi)), 0x1p-100f);
    } else {
        split(gp, g0, g1);
        g0f = g0.hi;
        g1f = g1.hi;
        lo = dl.hi;
        hi = dh.hi;
        mar = __fadd_rn(0x1p-43f * fabsf(qi.hi), 0x1p-100f);
    }
    T lim = T(1.0);
    if (P.limited && limit) {
        float nx[MJ], ny[MJ], nxk[H], nyk[H];
#pragma unroll
        for (int h = 0; h < H; h++) {
            if constexpr (is_fp64<T>) {
                nxk[h] = trunc_sat(ndk[h].x);
                nyk[h] = trunc_sat(ndk[h].y);
            } else {
                nxk[h] = ndk[h].x.hi;
                nyk[h] = ndk[h].y.hi;
            }
        }
#pragma unroll
        for (int j = 0; j < MJ; j++) {
            nx[j] = __shfl_sync(quad, nxk[j >> 2], j & 3, 4);
            ny[j] = __shfl_sync(quad, nyk[j >> 2], j & 3, 4);
        }
        bool low = false, unsure = false;
        const int j = limiting_neighbour<MJ>(mar, g0f, g1f, g0 == T(0.0) && g1 == T(0.0), lo, hi, dl == T(0.0),
                                             dh == T(0.0), nx, ny, UNI ? MJ : ne, low, unsure);
        if (unsure) {
            if constexpr (is_fp64<T>)
                lim = limit_exact(M, i, UNI ? MJ : ne, qin, k, qi, g0, g1);
            else
                lim = limit_exact(M, i, UNI ? MJ : ne, g0, g1, dl, dh);
        } else if (j >= 0) {
            const typename V2<T>::t nd = ld2<T>(M.g.s_nd, (size_t)j * Cs + i);
            if constexpr (is_fp64<T>) {
                const double dd = ebbsoft::mul(g0, nd.x) + ebbsoft::mul(g1, nd.y);
                const double s = soft_ratio(low ? dl : dh, dd, bad);
                lim = __double2hiint(s) < 0x3ff00000 ? s : 1.0;  // min(1, s), s >= -0
            } else {
                lim = fmin(lim, (low ? dl : dh) / sum(gp * pair(nd.x, nd.y)));
            }
        }
    }
    T lg0, lg1;
    if constexpr (is_fp64<T>) {
        lg0 = ebbsoft::mul(lim, g0);
        lg1 = ebbsoft::mul(lim, g1);
        ebbsoft::check<400>(lg0, bad);
        ebbsoft::check<400>(lg1, bad);
        if (__any_sync(quad, bad)) {
            if (k == 0) cell_plain<T, MJ, false>(M, P, A, st, i, ne, qin, limit);
            return;
        }
    } else {
        gp = both(lim) * gp;
    }
    if (P.need_grad) {
        typename V2<T>::t v;
        v.x = g0;
        v.y = g1;
        reinterpret_cast<typename V2<T>::t *>(A.grad)[4 * (size_t)i + k] = v;
    }
    if (A.lim) {  // limiter values, exported for ebb-reconstruct
        typename V2<T>::t v;
        v.x = lim;
        v.y = lim;
        reinterpret_cast<typename V2<T>::t *>(A.lim)[4 * (size_t)i + k] = v;
    }
    T *face = reinterpret_cast<T *>(A.face);
#pragma unroll
    for (int j = 0; j < MJ; j++) {
        if (UNI || j < ne) {
            const size_t s = (size_t)j * Cs + i;
            const typename V2<T>::t fd = slot(fdk, j);
            T f;
            if constexpr (is_fp64<T>) {
                f = qi + ebbsoft::mul(lg0, fd.x) + ebbsoft::mul(lg1, fd.y);
            } else {
                df x, y;
                split(gp * pair(fd.x, fd.y), x, y);
                f = qi + x + y;
            }
            if (pressure_negative4(f, k, quad)) {
                T l = fmin(T(1.0), shfl4(quad, lim, 0));
                l = fmin(l, shfl4(quad, lim, 1));
                l = fmin(l, shfl4(quad, lim, 2));
                l = fmin(l, shfl4(quad, lim, 3));
                f = qi + l * g0 * fd.x + l * g1 * fd.y;
            }
            face[4 * s + k] = f;
        }
    }
}

// One thread per cell: split precision, and the forms k_cell4 does not take.  Bound by the
// gathers' latency at the registers' limit on warps, so nothing here may cost a register
// of the split viscous form (80 of 85): its blocks run in ascending order only (a reversible
// order spills 40 bytes a thread instead of 16), the test for a stopped solve comes before
// the gathers, and the geometry takes plain loads; inviscid meshes, with registers to
// spare, mark it to leave L2 first (500,000 triangles 83.8 against 86.3 us a step; large ones
// do not, see shape_profile).  Measured
// so, per launch and step: 1M plate cells 47.9 -> 39.1 and 424 -> 409 us, 200,000 9.2 -> 8.6
// and 99.1 -> 98.2 us.
template <typename T, int MJ, bool LP, bool UNI, int PR>
__global__ void __launch_bounds__(cell_threads<T, PR>(), cell_minb<T, PR>())
    k_cell(const __grid_constant__ DMesh M, const __grid_constant__ DPhys P, const __grid_constant__ DArrays A,
           const T *__restrict__ qin, int limit)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const bool act = i < M.C;
    // read-only mesh data first, before the wait for the previous kernel.  Split path:
    // the neighbour rows are loaded whatever the cell's edge count (rows past it hold
    // 0), and the limiter's and the reconstruction's geometry (neighbour and face
    // midpoint offsets) is loaded here, not behind the gathers
    int ne = 0, inst = 0;
    CellPre<T, MJ> pre;
    if (act) {
        ne = UNI ? MJ : M.nedge[i];  // UNI: every cell has MJ edges (all triangles, all quads)
        if (M.cell_inst) inst = M.cell_inst[i];
        if constexpr (sizeof(T) == 4) {
            const int Cs = M.Cs;
            const auto geom = [](const void *p, size_t s) { return PR == 1 ? lds2<T>(p, s) : ld2<T>(p, s); };
#pragma unroll
            for (int j = 0; j < MJ; j++) {
                const int *p = M.s_nbr + (size_t)j * Cs + i;
                pre.nb[j] = PR == 1 ? stream(p) : *p;
            }
#pragma unroll
            for (int j = 0; j < MJ; j++) {
                pre.gm[j] = geom(M.g.s_gm, (size_t)j * Cs + i);
                pre.nd[j] = geom(M.g.s_nd, (size_t)j * Cs + i);
                pre.fd[j] = geom(M.g.s_fd, (size_t)j * Cs + i);
            }
        }
    }
    grid_dep_release();
    grid_dep_wait();
    if (!act) return;
    DState *st = A.st + inst;
    if (halted(st)) return;
    cell_body<T, MJ, LP>(M, P, A, st, i, UNI ? MJ : ne, qin, limit, pre);
}

template <typename T> __device__ __forceinline__ void load_grad(const void *grad, int c, T g[4][2])
{
    T a[4], b[4];
    const T *p = reinterpret_cast<const T *>(grad) + 8 * (size_t)c;
    ld4(p, a);
    ld4(p + 4, b);
    g[0][0] = a[0];
    g[0][1] = a[1];
    g[1][0] = a[2];
    g[1][1] = a[3];
    g[2][0] = b[0];
    g[2][1] = b[1];
    g[3][0] = b[2];
    g[3][1] = b[3];
}

template <typename T> __device__ __forceinline__ bool has_nan(const T F[4])
{
    return isnan(F[0]) || isnan(F[1]) || isnan(F[2]) || isnan(F[3]);
}

// The inviscid and viscous flux of a boundary face.  FP64: flux_soft.cuh's where the values
// allow it, with its quotients and roots on the integer pipe and its products on the FP64
// pipe (a third of the code).  A boundary block's latency is one face's, instruction
// fetches included: with device_math.cuh's ~450 FP64 instructions it was all of k_flux on
// small meshes (a step of 1024 quads 69 us; 67 us with every product on the integer pipe;
// so, 62 us).
template <typename T>
__device__ __noinline__ void inviscid_plain(int kind, const T qL[4], const T qR[4], T nx, T ny, T F[4], T &sMax)
{
    inviscid_flux(kind, qL, qR, nx, ny, F, sMax);
}
template <typename T>
__device__ __noinline__ void viscous_plain(const ViscConst<T> &vc, T mu, const T q[4], const T dq[4][2], T nx, T ny, T F[4])
{
    diffusive_flux(vc, mu, q, dq, nx, ny, F);
}
template <typename T>
__device__ __forceinline__ void face_inviscid(const DMesh &M, int kind, const T qL[4], const T qR[4], T nx, T ny, T F[4],
                                              T &sMax)
{
    if constexpr (is_fp64<T>) {
        bool bad = !M.soft;
        double X[4], s;
        inviscid_flux2_soft<false>(kind, qL, qR, nx, ny, X, s, bad);
        if (bad) {
            const double a[4] = {qL[0], qL[1], qL[2], qL[3]}, b[4] = {qR[0], qR[1], qR[2], qR[3]};
            inviscid_plain<T>(kind, a, b, nx, ny, X, s);
        }
        sMax = s;
#pragma unroll
        for (int k = 0; k < 4; k++) F[k] = bad ? X[k] : 0.5 * X[k];
    } else {
        inviscid_flux(kind, qL, qR, nx, ny, F, sMax);
    }
}
template <typename T>
__device__ __forceinline__ void face_viscous(const DMesh &M, const ViscConst<T> &vc, T mu, const T q[4], const T dq[4][2],
                                             T nx, T ny, T F[4])
{
    if constexpr (is_fp64<T>) {
        bool bad = !M.soft;
        ebbsoft::check<60>(q[0], bad);
        bad |= !ebbsoft::divisor_ok(q[0]);
#pragma unroll
        for (int k = 1; k < 4; k++) ebbsoft::check<100>(q[k], bad);
        double X[4];
        diffusive_flux2_soft<false>(vc, mu, q, dq, nx, ny, X, bad);
        if (bad) {
            const double a[4] = {q[0], q[1], q[2], q[3]};
            const double g[4][2] = {{dq[0][0], dq[0][1]}, {dq[1][0], dq[1][1]}, {dq[2][0], dq[2][1]}, {dq[3][0], dq[3][1]}};
            viscous_plain<T>(vc, mu, a, g, nx, ny, X);
        }
        F[0] = zero_dot(nx, ny);
#pragma unroll
        for (int k = 1; k < 4; k++) F[k] = bad ? X[k] : 0.5 * X[k];
    } else {
        diffusive_flux(vc, mu, q, dq, nx, ny, F);
    }
}

template <typename T>
__device__ __forceinline__ void boundary_flux(const DMesh &M, const DPhys &P, const DArrays &A, const T *qin, int b)
{
    const T G = K<T>::g;
    const int type = M.b_type[b];
    const size_t fsl = (size_t)M.b_slot[b];
    T qL[4];
    ld4(reinterpret_cast<const T *>(A.face) + 4 * fsl, qL);
    const typename V2<T>::t n = ld2<T>(M.g.b_n, b);
    const T nx = n.x, ny = n.y;
    T F[4], sMax = 0;
    const int owner = M.b_cell[b];
    const int ghost = M.C + b;
    const int inst = M.cell_inst ? M.cell_inst[owner] : 0;
    DState *st = A.st + inst;
    if (halted(st)) return;
    const ViscConst<T> pr = visc_const<T>(P);
    const T mu = visc_mu<T>(M, P, inst);
    switch (type & 0xff) {
    case BC_DIRICHLET:
    case BC_FULLSTATE: {
        T qR[4];
        ld4(ptr<T>((type & 0xff) == BC_DIRICHLET ? M.g.b_dmid : M.g.b_data) + 4 * (size_t)b, qR);
        face_inviscid(M, P.flux, qL, qR, nx, ny, F, sMax);
        if (P.viscous) {
            T g1[4][2], g2[4][2], dq[4][2], qa[4], Fv[4];
            load_grad<T>(A.grad, owner, g1);
            load_grad<T>(A.grad, ghost, g2);
            for (int k = 0; k < 4; k++) {
                qa[k] = half(qL[k] + qR[k]);
                dq[k][0] = half(g1[k][0] + g2[k][0]);
                dq[k][1] = half(g1[k][1] + g2[k][1]);
            }
            face_viscous(M, pr, mu, qa, dq, nx, ny, Fv);
            for (int k = 0; k < 4; k++) F[k] = F[k] - Fv[k];
        }
        break;
    }
    case BC_INVWALL: {
        T inv = ratio(T(1), qL[0]);
        T vp0 = inv * qL[1], vp1 = inv * qL[2];
        T vn = vp0 * nx + vp1 * ny;
        T t0 = vp0 - vn * nx, t1 = vp1 - vn * ny;
        T vel = root(t0 * t0 + t1 * t1);
        T p = (G - 1) * (qL[3] - T(0.5) * qL[0] * (vel * vel));
        T a = root(G * ratio(p, qL[0]));
        if (p < 0) p = T(1.0e-12);
        F[0] = 0;
        F[1] = p * nx;
        F[2] = p * ny;
        F[3] = 0;
        sMax = fabs(a);
        break;
    }
    case BC_VISCWALL: {
        T vel = 0.0;
        T p = (G - 1) * (qL[3] - T(0.5) * qL[0] * (vel * vel));
        T a = root(G * ratio(p, qL[0]));
        if (p < 0) p = T(1.0e-12);
        T qR[4] = {qL[0], qL[1] * -1, qL[2] * -1, qL[3]};
        T qa[4], dq[4][2], Fv[4];
        for (int k = 0; k < 4; k++) qa[k] = half(qL[k] + qR[k]);
        qa[1] = 0.0;
        qa[2] = 0.0;
        load_grad<T>(A.grad, owner, dq);
        const T e = ratio(qa[3], qa[0]);
        dq[3][0] = e * dq[0][0];
        dq[3][1] = e * dq[0][1];
        face_viscous(M, pr, mu, qa, dq, nx, ny, Fv);
        F[0] = 0 - Fv[0];
        F[1] = p * nx - Fv[1];
        F[2] = p * ny - Fv[2];
        F[3] = 0 - Fv[3];
        sMax = fabs(a);
        break;
    }
    case BC_CONSTP: {
        T qg[4];
        ld4(qin + 4 * (size_t)ghost, qg);
        T p = pressure(qg);
        T u = ratio(qg[1], qg[0]), v = ratio(qg[2], qg[0]);
        T a = root(G * ratio(p, qg[0]));
        convective_flux(p, u, v, qg[0], qg[3], nx, ny, F);
        sMax = fabs(a);
        break;
    }
    case BC_SYMMETRY: {
        T v0 = ratio(qL[1], qL[0]), v1 = ratio(qL[2], qL[0]), n0, n1;
        reflect(type, ptr<T>(M.g.b_refl) + 4 * (size_t)b, v0, v1, n0, n1);
        T qR[4] = {qL[0], qL[0] * n0, qL[0] * n1, qL[3]};
        face_inviscid(M, P.flux, qL, qR, nx, ny, F, sMax);
        if (P.viscous) {
            T gp[4][2], qa[4], Fv[4];
            load_grad<T>(A.grad, owner, gp);
            for (int k = 0; k < 4; k++) qa[k] = half(qL[k] + qR[k]);
            // bGrad = gradp*nOuter + (A*gradp)*(I - 2 nOuter), solve.d:913-925
            T nO[2][2] = {{nx * nx, nx * ny}, {ny * nx, ny * ny}};
            T Am[4][4] = {{1, 0, 0, 0}, {0, 1 - nO[0][0], 0 - nO[0][1], 0}, {0, 0 - nO[1][0], 1 - nO[1][1], 0},
                          {0, 0, 0, 1}};
            T t2[2][2] = {{1 - 2 * nO[0][0], 0 - 2 * nO[0][1]}, {0 - 2 * nO[1][0], 1 - 2 * nO[1][1]}};
            T t1[4][2], bG[4][2];
            for (int r = 0; r < 4; r++)
                for (int c = 0; c < 2; c++) {
                    T acc = 0.0;
                    for (int k = 0; k < 4; k++) acc += Am[r][k] * gp[k][c];
                    t1[r][c] = acc;
                }
            for (int r = 0; r < 4; r++)
                for (int c = 0; c < 2; c++) {
                    T a3 = 0.0;
                    for (int k = 0; k < 2; k++) a3 += t1[r][k] * t2[k][c];
                    T a1 = 0.0;
                    for (int k = 0; k < 2; k++) a1 += gp[r][k] * nO[k][c];
                    bG[r][c] = a1 + a3;
                }
            face_viscous(M, pr, mu, qa, bG, nx, ny, Fv);
            for (int k = 0; k < 4; k++) F[k] = F[k] - Fv[k];
        }
        break;
    }
    case BC_TPINFLOW: {
        T qR[4];
        ld4(qin + 4 * (size_t)ghost, qR);
        face_inviscid(M, P.flux, qL, qR, nx, ny, F, sMax);
        if (P.viscous) {
            T gp[4][2], qa[4], Fv[4];
            load_grad<T>(A.grad, owner, gp);
            for (int k = 0; k < 4; k++) qa[k] = half(qL[k] + qR[k]);
            face_viscous(M, pr, mu, qa, gp, nx, ny, Fv);
            for (int k = 0; k < 4; k++) F[k] = F[k] - Fv[k];
        }
        break;
    }
    default:
        F[0] = F[1] = F[2] = F[3] = T(NAN);
    }
    if (has_nan(F)) flag_error(st, 1, ERR_NAN_EDGE, (unsigned)M.b_ref[b]);
    const T len = ld1<T>(M.g.b_len, b);
    const size_t e = (size_t)M.Eint + b;
    T lf[4] = {len * F[0], len * F[1], len * F[2], len * F[3]};
    st4(reinterpret_cast<T *>(A.fl) + 4 * e, lf);
    if (M.speeds) reinterpret_cast<T *>(A.fs)[e] = len * sMax;
}

// FP64 and double-float: a call, so that the interior faces' registers and code are theirs
// alone (500,000 plate cells, double-float: step 827 -> 786 us; split precision is 1 to 5%
// faster with it in line)
template <typename T>
__device__ __noinline__ void boundary_flux_call(const DMesh &M, const DPhys &P, const DArrays &A, const T *qin, int b)
{
    boundary_flux<T>(M, P, A, qin, b);
}

// len * flux and len * sMax of interior edge e from its two face states (and, viscous,
// its cells' gradients)
template <typename T>
__device__ __forceinline__ void edge_flux(const DMesh &M, const DPhys &P, const DArrays &A, DState *st, int inst, int e,
                                          int2 sl, typename V2<T>::t n, T len, const T qL[4], const T qR[4])
{
    T F[4], sMax;
    inviscid_flux(P.flux, qL, qR, n.x, n.y, F, sMax);
    if (P.viscous) {
        const int2 c = make_int2(slot_cell(M, sl.x), slot_cell(M, sl.y));
        T g1[4][2], g2[4][2], dq[4][2], qa[4], Fv[4];
        load_grad<T>(A.grad, c.x, g1);
        load_grad<T>(A.grad, c.y, g2);
        for (int k = 0; k < 4; k++) {
            qa[k] = half(qL[k] + qR[k]);
            dq[k][0] = half(g1[k][0] + g2[k][0]);
            dq[k][1] = half(g1[k][1] + g2[k][1]);
        }
        diffusive_flux(visc_const<T>(P), visc_mu<T>(M, P, inst), qa, dq, n.x, n.y, Fv);
        for (int k = 0; k < 4; k++) F[k] = F[k] - Fv[k];
    }
    if (has_nan(F)) flag_error(st, 2, ERR_NAN_EDGE, (unsigned)M.e_ref[e]);
    T lf[4] = {len * F[0], len * F[1], len * F[2], len * F[3]};
    st4(reinterpret_cast<T *>(A.fl) + 4 * (size_t)e, lf);
    if (M.speeds) reinterpret_cast<T *>(A.fs)[e] = len * sMax;
}

// edge_flux in double-float with flux_df.cuh's packed arithmetic
__device__ __forceinline__ void edge_flux_df(const DMesh &M, const DPhys &P, const DArrays &A, DState *st, int inst, int e,
                                             int2 sl, df2 n, df len, const df qL[4], const df qR[4])
{
    df sMax;
    dfp F03, F12;
    if (P.flux == 1)
        roe_flux_df(qL, qR, n.x, n.y, F03, F12, sMax);
    else
        rusanov_flux_df(qL, qR, n.x, n.y, F03, F12, sMax);
    if (P.viscous) {
        const int2 c = make_int2(slot_cell(M, sl.x), slot_cell(M, sl.y));
        df g1[4][2], g2[4][2], qa[4], o3;
        dfp dq[4], o12;
        load_grad<df>(A.grad, c.x, g1);
        load_grad<df>(A.grad, c.y, g2);
#pragma unroll
        for (int k = 0; k < 4; k++) dq[k] = half(pair(g1[k][0], g1[k][1]) + pair(g2[k][0], g2[k][1]));
        split(half(pair(qL[0], qL[1]) + pair(qR[0], qR[1])), qa[0], qa[1]);
        split(half(pair(qL[2], qL[3]) + pair(qR[2], qR[3])), qa[2], qa[3]);
        diffusive_flux_df(visc_const<df>(P), visc_mu<df>(M, P, inst), qa, dq, n.x, n.y, o3, o12);
        F03 = F03 - pair(df(0.0f), o3);
        F12 = F12 - o12;
    }
    const dfp l = both(len), a = l * F03, b = l * F12;
    df f[4];
    split(a, f[0], f[3]);
    split(b, f[1], f[2]);
    if (has_nan(f)) flag_error(st, 2, ERR_NAN_EDGE, (unsigned)M.e_ref[e]);
    st4(reinterpret_cast<df *>(A.fl) + 4 * (size_t)e, f);
    if (M.speeds) reinterpret_cast<df *>(A.fs)[e] = len * sMax;
}

// plain FP64: the edges edge_flux_soft leaves
template <typename T>
__device__ __noinline__ void edge_flux_plain(const DMesh &M, const DPhys &P, const DArrays &A, DState *st, int inst, int e)
{
    const int2 sl = reinterpret_cast<const int2 *>(M.e_slot)[e];
    T qL[4], qR[4];
    ld4(reinterpret_cast<const T *>(A.face) + 4 * (size_t)sl.x, qL);
    ld4(reinterpret_cast<const T *>(A.face) + 4 * (size_t)sl.y, qR);
    edge_flux<T>(M, P, A, st, inst, e, sl, ld2<T>(M.g.e_n, e), ld1<T>(M.g.e_len, e), qL, qR);
}

// edge_flux in FP64 with flux_soft.cuh's arithmetic; false (and nothing written) where
// that does not hold for the edge's values.  No value here is a NaN.
__device__ __forceinline__ bool edge_flux_soft(const DMesh &M, const DPhys &P, const DArrays &A, int inst, int e, int2 sl,
                                               double2 n, double len, double qL[4], const double qR[4])
{
    double F[4], sMax;  // F: twice the flux
    bool bad = false;
    inviscid_flux2_soft<true>(P.flux, qL, qR, n.x, n.y, F, sMax, bad);
    if (P.viscous) {
        const int2 c = make_int2(slot_cell(M, sl.x), slot_cell(M, sl.y));
        double g1[4][2], g2[4][2], Fv[4];
        load_grad<double>(A.grad, c.x, g1);
        load_grad<double>(A.grad, c.y, g2);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            qL[k] = qL[k] + qR[k];
            g1[k][0] = g1[k][0] + g2[k][0];
            g1[k][1] = g1[k][1] + g2[k][1];
        }
        diffusive_flux2_soft<true>(visc_const<double>(P), visc_mu<double>(M, P, inst), qL, g1, n.x, n.y, Fv, bad);
        F[0] = F[0] - zero_dot(n.x, n.y);
#pragma unroll
        for (int k = 1; k < 4; k++) F[k] = F[k] - Fv[k];
    }
    if (bad) return false;
    const double hl = 0.5 * len;
    const double lf[4] = {hl * F[0], hl * F[1], hl * F[2], hl * F[3]};
    st4(reinterpret_cast<double *>(A.fl) + 4 * (size_t)e, lf);
    if (M.speeds) reinterpret_cast<double *>(A.fs)[e] = len * sMax;
    return true;
}

template <typename T, int PR>
__global__ void __launch_bounds__(flux_threads<T, PR>(), flux_minb<T, PR>())
    k_flux(const __grid_constant__ DMesh M, const __grid_constant__ DPhys P, const __grid_constant__ DArrays A,
           const T *__restrict__ qin, int nbb)
{
    // the boundary blocks first: theirs is the longest latency
    if ((int)blockIdx.x < nbb) {
        grid_dep_release();
        grid_dep_wait();
        const int b = blockIdx.x * blockDim.x + threadIdx.x;
        if (b < M.G) {
            if constexpr (is_fp32<T>)
                boundary_flux<T>(M, P, A, qin, b);
            else
                boundary_flux_call<T>(M, P, A, qin, b);
        }
        return;
    }
    const int nbi = gridDim.x - nbb, blk = (int)blockIdx.x - nbb;
    const int e = (M.rev ? nbi - 1 - blk : blk) * blockDim.x + threadIdx.x;
    const bool act = e < M.Eint;
    // read-only mesh data before the wait for the previous kernel
    int inst = 0;
    int2 sl = make_int2(0, 0);
    typename V2<T>::t n = {};
    T len = T(0.0);
    if (act) {
        sl = stream(reinterpret_cast<const int2 *>(M.e_slot) + e);
        if (M.cell_inst) inst = M.cell_inst[slot_cell(M, sl.x)];
        n = ld2<T>(M.g.e_n, e);
        len = ld1<T>(M.g.e_len, e);
    }
    grid_dep_release();
    grid_dep_wait();
    if (!act) return;
    DState *st = A.st + inst;
    T qL[4], qR[4];
    ld4(reinterpret_cast<const T *>(A.face) + 4 * (size_t)sl.x, qL);
    ld4(reinterpret_cast<const T *>(A.face) + 4 * (size_t)sl.y, qR);
    if (halted(st)) return;  // behind the gathers: they and this test wait together
    if constexpr (is_fp64<T>) {
        if (!(M.soft && edge_flux_soft(M, P, A, inst, e, sl, n, len, qL, qR))) edge_flux_plain<T>(M, P, A, st, inst, e);
    } else if constexpr (is_df<T>) {
        edge_flux_df(M, P, A, st, inst, e, sl, n, len, qL, qR);
    } else {
        edge_flux<T>(M, P, A, st, inst, e, sl, n, len, qL, qR);
    }
}

// ---- fixed-order block reductions -------------------------------------------
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double warp_min(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_max(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_sumf(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = v + __shfl_down_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ float warp_minf(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fminf(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ float warp_maxf(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// o = a b for four values.  FP64: on the integer pipe where the values allow it (the
// plain update kernel is bound by the FP64 pipe like the others: 76% busy, with 10% of
// the issue slots used).
template <typename T> __device__ __forceinline__ void mul4(const T a[4], T b, T o[4])
{
#pragma unroll
    for (int k = 0; k < 4; k++) o[k] = a[k] * b;
}
template <> __device__ __forceinline__ void mul4<double>(const double a[4], double b, double o[4])
{
    bool bad = false;
    ebbsoft::check<400>(b, bad);
#pragma unroll
    for (int k = 0; k < 4; k++) ebbsoft::check<400>(a[k], bad);
    if (bad) {
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = a[k] * b;
    } else {
#pragma unroll
        for (int k = 0; k < 4; k++) o[k] = ebbsoft::mul(a[k], b);
    }
}
// x with its sign changed where bit 31 of s is set.  (Two branches, one with -x, ran both
// in nearly every warp: edges of either orientation alternate from cell to cell.)
__device__ __forceinline__ float flip(float x, int s) { return __int_as_float(__float_as_int(x) ^ (s & 0x80000000)); }
__device__ __forceinline__ double flip(double x, int s)
{
    return __hiloint2double(__double2hiint(x) ^ (s & 0x80000000), __double2loint(x));
}
__device__ __forceinline__ df flip(df x, int s) { return df(flip(x.hi, s), flip(x.lo, s)); }
// acc + 2 x (2 x is exact: one rounding)
template <typename T> __device__ __forceinline__ T plus_twice(T acc, T x) { return acc + T(2.0) * x; }
template <> __device__ __forceinline__ double plus_twice<double>(double acc, double x) { return fma(2.0, x, acc); }
// the larger of m and |x| for m >= 0; a NaN x leaves m
__device__ __forceinline__ double max_abs(double m, double x)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
    const unsigned long long c = (unsigned long long)__double_as_longlong(m);
    return b > c && b <= 0x7ff0000000000000ull ? __longlong_as_double((long long)b) : m;
}

// Residual of one interior cell and the stage combination.  The solution's update runs
// in FP64 for every precision form.  FP64 path: qin/qout are double stage states as in
// integrators.d.  Split path: qin is the FP32 stage input, q64 is updated in FP64 and
// the next stage input (qout) is its FP32 rounding.  Double-float path: stages before
// the last form their stage state in double-float from the solution's double-float
// copy; the last updates q64 in FP64 and refreshes that copy.
template <typename T, int ST, int MJ, bool UNI, int PR>
__global__ void __launch_bounds__(UPD_THREADS, upd_minb<T, PR>()) k_update(DMesh M, DPhys P, DArrays A, const T *__restrict__ qin, T *qout,
                                                       int dt_update, int need_dt, int final_stage)
{
    constexpr bool SPLIT = sizeof(T) == 4;
    constexpr bool LARGE = PR == 2;  // loads where they are used, 32 registers: shape_profile
    const int blk = LARGE ? (int)blockIdx.x : ordered_block(M, gridDim.x);
    int i, iend, inst = 0;
    if (M.blk_first) {  // batched arena: each block lies inside one instance's cell range
        i = M.blk_first[blk] + threadIdx.x;
        iend = M.blk_end[blk];
        inst = M.blk_inst[blk];
    } else {
        i = blk * blockDim.x + threadIdx.x;
        iend = M.C;
    }
    const bool act = i < iend;
    const int Cs = M.Cs;
    const bool speeds = need_dt || (P.local_ts && dt_update);  // the edges' wave speeds are read
    // read-only mesh data before the wait for the previous kernel: every edge row is
    // loaded whatever the cell's edge count (rows past it hold 0)
    int ev[MJ], ne = 0;
    typename V2<T>::t sn[MJ];  // split path: the edges' normals and lengths
    T sl[MJ], nia = T(0.0), perim = T(1.0), dlen = T(0.0);
    if (act) {
#pragma unroll
        for (int j = 0; j < MJ; j++) ev[j] = stream(M.s_edge + (size_t)j * Cs + i);
        ne = UNI ? MJ : M.nedge[i];
        if (!LARGE) {
            nia = ld1<T>(M.g.neg_inv_area, i);
            if (speeds) {
                perim = ld1<T>(M.g.perim, i);
                dlen = ld1<T>(M.g.dlen, i);
            }
        }
        if constexpr (SPLIT) {
#pragma unroll
            for (int j = 0; j < MJ; j++) {
                sn[j] = ld2<T>(M.g.e_n, (size_t)(ev[j] & 0x7fffffff));
                sl[j] = ld1<T>(M.g.e_len, (size_t)(ev[j] & 0x7fffffff));
            }
        }
    }
    grid_dep_release();
    grid_dep_wait();
    DState *st = A.st + inst;
    constexpr bool AUX = ST == ST_RK2_2 || (SPLIT && ST == ST_TVD_2) || ST == ST_RK4_2 || ST == ST_RK4_3 || ST == ST_RK4_4;
    T *aux = reinterpret_cast<T *>(A.aux);
    T f[MJ][4], fe[MJ], ax[4], qb[4];
    double q0[4];
    auto gather = [&]() {
        const T *fl = reinterpret_cast<const T *>(A.fl);
        const T *fs = reinterpret_cast<const T *>(A.fs);
#pragma unroll
        for (int j = 0; j < MJ; j++) {
            if (j < ne) {
                const size_t e = (size_t)(ev[j] & 0x7fffffff);
                ld4(fl + 4 * e, f[j]);
                fe[j] = speeds ? fs[e] : T(0.0);
            }
        }
    };
    if (!LARGE && act) gather();
    // the solution and the earlier stages, loaded where they are used: held from here on
    // with the flux gathers, they spill (1M plate cells, split: step 450 instead of 433 us)
    auto stage_loads = [&]() {
        if constexpr (AUX) ld4(aux + 4 * (size_t)i, ax);
        if constexpr (ST != ST_RESID) {
            if (!is_fp64<T> && !final_stage)
                ld4(reinterpret_cast<const T *>(A.qs1) + 4 * (size_t)i, qb);
            else
                ld4(A.q64 + 4 * (size_t)i, q0);
        }
    };
    if (halted(st)) return;
    double dtc = INFINITY, rm = 0.0;
    double ss[4] = {0, 0, 0, 0}, vs[4] = {0, 0, 0, 0};
    float fss[4] = {0, 0, 0, 0}, fvs[4] = {0, 0, 0, 0};  // split path: FP32 lane values
    float fdtc = INFINITY, frm = 0.0f;
    bool bad = false;
    if (act) {
        if (LARGE) gather();
        // the sums add in edge order
        T r[4] = {T(0.0), T(0.0), T(0.0), T(0.0)};
        T sAve = 0;
#pragma unroll
        for (int j = 0; j < MJ; j++) {
            if (j < ne) {
                if (is_fp64<T> && j == 0) {  // 0 + x without the FP64 pipe
#pragma unroll
                    for (int k = 0; k < 4; k++) r[k] = zero_plus(flip(f[0][k], ev[0]));
                    sAve = fe[0];
                    continue;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) r[k] = r[k] + flip(f[j][k], ev[j]);
                sAve += fe[j];
            }
        }
        if constexpr (SPLIT) {
            // Freestream preservation.  Subtract the same edge sum of the cell's own
            // physical flux, sum_j m_j len_j F(q_i).n_j = F(q_i) . sum_j m_j len_j n_j,
            // which is zero but for the rounding of the FP32 edge terms.  Where the
            // cell and its neighbours hold one state (face states equal to it, the flux
            // of two equal states equal to the physical flux, computed without
            // contraction in both kernels) both sums are the same bits and the residual
            // is exactly zero, as in FP64; otherwise the correction is of the size of
            // the FP32 rounding.  Without it a uniform region takes FP32-rounding-size
            // increments every step, which seed the locally unstable modes the scheme
            // has on some meshes (a plain FP64 run with 1e-7 noise added each step
            // fails at the same edge as the split run).  It runs on every cell: limited
            // to cells whose neighbours hold bitwise their state, 13 of 512 batch
            // instances failed instead of 6 (nearly uniform cells then take the full
            // edge-term rounding); limited to neighbours within 1e-3, the failures and
            // the accuracy were those of the ungated form, at a higher cost.
            T qc[4];
            ld4(qin + 4 * (size_t)i, qc);
            const T uc = qc[1] / qc[0], vc = qc[2] / qc[0];
            const T pc = pressure_of(qc[0], uc, vc, qc[3]);
            T c[4] = {T(0.0), T(0.0), T(0.0), T(0.0)};
#pragma unroll
            for (int j = 0; j < MJ; j++) {
                if (j < ne) {
                    const T len = flip(sl[j], ev[j]);
                    T F[4];
                    convective_flux(pc, uc, vc, qc[0], qc[3], sn[j].x, sn[j].y, F);
                    // len F rounded on its own, as k_flux stores it (no contraction)
#pragma unroll
                    for (int k = 0; k < 4; k++) c[k] = __fadd_rn(c[k], __fmul_rn(len, F[k]));
                }
            }
#pragma unroll
            for (int k = 0; k < 4; k++) r[k] = r[k] - c[k];
        }
        T *cdt = reinterpret_cast<T *>(A.cdt);
        if (speeds) {
            if (LARGE) {
                perim = ld1<T>(M.g.perim, i);
                dlen = ld1<T>(M.g.dlen, i);
            }
            sAve = ratio(sAve, perim);
            T c = ratio(cfl_of<T>(st) * dlen, sAve);
            if (need_dt) {
                if (SPLIT)
                    fdtc = (float)c;
                else
                    dtc = to_f64(c);
            }
            if (P.local_ts && dt_update) cdt[i] = isnan(c) ? T(0.0) : c;
        }
        if (SPLIT) {
#pragma unroll
            for (int k = 0; k < 4; k++)
                if ((float)fabs(r[k]) > frm) frm = (float)fabs(r[k]);
        } else if constexpr (is_df<T>) {  // the largest |r| found in double-float, one conversion
            T m = T(0.0f);
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (fabs(r[k]) > m) m = fabs(r[k]);
            rm = to_f64(m);
        } else {
#pragma unroll
            for (int k = 0; k < 4; k++) rm = max_abs(rm, r[k]);
        }
        if (!LARGE) stage_loads();
        T R[4];
        if (LARGE) nia = ld1<T>(M.g.neg_inv_area, i);
        mul4(r, nia, R);
        if (LARGE) stage_loads();
        if (P.mms) {
            T S[4];
            ld4(ptr<T>(M.g.src) + 4 * (size_t)i, S);
#pragma unroll
            for (int k = 0; k < 4; k++) R[k] = R[k] + S[k];
        }
        if (ST == ST_RESID) {
            st4(reinterpret_cast<T *>(A.R) + 4 * (size_t)i, R);
        } else if constexpr (SPLIT) {
            // increments at the precision of R.  Intermediate stage inputs are FP32
            // (the FP32 shadow of the solution plus the increment); the final stage
            // accumulates the solution u += inc in FP64 and refreshes the shadow.
            const float dtf = st->dtf, hf = P.local_ts ? (float)cdt[i] : dtf;
            float inc[4];
            if (ST == ST_EULER || ST == ST_TVD_1) {
                if (ST == ST_TVD_1) st4(aux + 4 * (size_t)i, R);
#pragma unroll
                for (int k = 0; k < 4; k++) inc[k] = hf * R[k];
            } else if (ST == ST_RK2_1) {
                st4(aux + 4 * (size_t)i, R);
#pragma unroll
                for (int k = 0; k < 4; k++) inc[k] = dtf * R[k];
            } else if (ST == ST_RK2_2) {
                const float hh = P.local_ts ? hf * 0.5f : st->dt_half_f;
#pragma unroll
                for (int k = 0; k < 4; k++) inc[k] = hh * (ax[k] + R[k]);
            } else if (ST == ST_TVD_2) {  // 0.5 (q + (q + h R1) + h R2) = q + 0.5 h (R1 + R2)
#pragma unroll
                for (int k = 0; k < 4; k++) inc[k] = (0.5f * hf) * (ax[k] + R[k]);
            } else if (ST == ST_RK4_1) {
                st4(aux + 4 * (size_t)i, R);
#pragma unroll
                for (int k = 0; k < 4; k++) inc[k] = st->dt_half_f * R[k];
            } else if (ST == ST_RK4_2 || ST == ST_RK4_3) {
#pragma unroll
                for (int k = 0; k < 4; k++) ax[k] = ax[k] + 2.0f * R[k];
                st4(aux + 4 * (size_t)i, ax);
                const float h2 = ST == ST_RK4_2 ? st->dt_half_f : dtf;
#pragma unroll
                for (int k = 0; k < 4; k++) inc[k] = h2 * R[k];
            } else {  // ST_RK4_4
                const float hh = P.local_ts ? hf / 6.0f : st->dt_sixth_f;
#pragma unroll
                for (int k = 0; k < 4; k++) inc[k] = hh * (ax[k] + R[k]);
            }
            T o[4];
            if (final_stage) {
                // u += inc in FP64; the conversions run on the integer pipe (an FP64
                // conversion costs about as much FP64-pipe time as the add)
                double out[4];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    out[k] = q0[k] + f2d_int(inc[k]);
                    o[k] = d2f_int(out[k]);
                }
                st4(A.q64 + 4 * (size_t)i, out);
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    fss[k] = inc[k] * inc[k];
                    fvs[k] = o[k];
                }
                bad = isnan(o[0]) || isnan(o[1]) || isnan(o[2]) || isnan(o[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) o[k] = qb[k] + inc[k];
            }
            st4(qout + 4 * (size_t)i, o);
        } else if (is_df<T> && !final_stage) {
            // double-float, a stage before the last: the stage state is the solution's
            // double-float copy plus the stage increment, all in double-float (it is
            // stored as one anyway); the FP64 solution is updated by the last stage
            if constexpr (is_df<T> && (ST == ST_RK2_1 || ST == ST_TVD_1 || ST == ST_RK4_1 || ST == ST_RK4_2 ||
                                       ST == ST_RK4_3)) {
                    T h = st->dtw;
                if (ST == ST_TVD_1) {
                    if (P.local_ts) h = cdt[i];
                } else if (ST == ST_RK2_1 || ST == ST_RK4_1) {
                    st4(aux + 4 * (size_t)i, R);
                    if (ST == ST_RK4_1) h = st->dt_half_w;
                } else {
#pragma unroll
                    for (int k = 0; k < 4; k++) ax[k] = ax[k] + T(2.0f) * R[k];
                    st4(aux + 4 * (size_t)i, ax);
                    if (ST == ST_RK4_2) h = st->dt_half_w;
                }
                T o[4];
#pragma unroll
                for (int k = 0; k < 4; k++) o[k] = qb[k] + h * R[k];
                st4(qout + 4 * (size_t)i, o);
            }
        } else {
            double Rd[4], out[4];
#pragma unroll
            for (int k = 0; k < 4; k++) Rd[k] = to_f64(R[k]);
            const double dt = st->dt;
            const double h = P.local_ts ? to_f64(cdt[i]) : dt;
            double x[4], f = h, inc[4];  // the stage's increment is f x
#pragma unroll
            for (int k = 0; k < 4; k++) x[k] = Rd[k];
            if (ST == ST_RK2_1) {
                st4(aux + 4 * (size_t)i, R);
                f = dt;
            } else if (ST == ST_RK2_2) {
#pragma unroll
                for (int k = 0; k < 4; k++) x[k] = to_f64(ax[k] + R[k]);
                f = P.local_ts ? h / 2.0 : st->dt_half;
            } else if (ST == ST_RK4_1) {
                st4(aux + 4 * (size_t)i, R);
                f = st->dt_half;
            } else if (ST == ST_RK4_2 || ST == ST_RK4_3) {
#pragma unroll
                for (int k = 0; k < 4; k++) ax[k] = plus_twice(ax[k], R[k]);
                st4(aux + 4 * (size_t)i, ax);
                f = ST == ST_RK4_2 ? st->dt_half : dt;
            } else if (ST == ST_RK4_4) {
#pragma unroll
                for (int k = 0; k < 4; k++) x[k] = to_f64(ax[k] + R[k]);
                f = P.local_ts ? ratio(h, 6.0) : st->dt_sixth;
            }
            if constexpr (is_fp64<T>) mul4(x, f, inc);
            T qf[4];
            if (ST == ST_TVD_2) ld4(qin + 4 * (size_t)i, qf);
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double b = ST == ST_TVD_2 ? q0[k] + to_f64(qf[k]) : q0[k];
                // the reference's two roundings on the plain path, one on the double-float path
                out[k] = is_fp64<T> ? b + inc[k] : fma(f, x[k], b);
                if (ST == ST_TVD_2) out[k] = half(out[k]);
            }
            if (final_stage) {
                st4(A.q64 + 4 * (size_t)i, out);
                if (!is_fp64<T>) {  // the double-float shadow of the solution
                    T o[4] = {from_f64<T>(out[0]), from_f64<T>(out[1]), from_f64<T>(out[2]), from_f64<T>(out[3])};
                    st4(qout + 4 * (size_t)i, o);
                }
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    double d = out[k] - q0[k];
                    ss[k] = d * d;
                    vs[k] = out[k];
                }
                bad = isnan(out[0]) || isnan(out[1]) || isnan(out[2]) || isnan(out[3]);
            } else {
                T o[4] = {from_f64<T>(out[0]), from_f64<T>(out[1]), from_f64<T>(out[2]), from_f64<T>(out[3])};
                st4(qout + 4 * (size_t)i, o);
            }
        }
    }
    if (bad) flag_error(st, 3, ERR_NAN_CELL, (unsigned)M.cell_ref[i]);
    // block reductions: dt (min), Rmax (max), RMS partials (sum) in a fixed tree
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (SPLIT) {
        // The whole block in FP32 (an FP64 instruction costs a warp the same with one
        // lane active as with 32), one conversion per block value; the grid-wide
        // accumulation of the block partials is FP64.  Every thread's values go to
        // shared memory and one warp reduces each column (lane l takes rows l, l+32,
        // ..., then a shuffle tree): 10 values cost a warp ~60 instructions instead of
        // ten 5-level shuffle trees.  Column 1 holds -Rmax so that columns 0 and 1 are
        // both minima.  Fixed order.
        constexpr int WF = 11;  // row stride in floats: conflict-free column reads
        __shared__ float shf[UPD_THREADS * WF];
        __shared__ float partf[10];
        const int t = threadIdx.x;
        const int ncol = final_stage ? 10 : 2;
        shf[t * WF + 0] = fdtc;
        shf[t * WF + 1] = -frm;
        if (final_stage) {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                shf[t * WF + 2 + k] = fss[k];
                shf[t * WF + 6 + k] = fvs[k];
            }
        }
        __syncthreads();
        for (int c = w; c < ncol; c += UPD_THREADS / 32) {
            float a = shf[lane * WF + c];
            if (c < 2) {
#pragma unroll
                for (int r = 1; r < UPD_THREADS / 32; r++) a = fminf(a, shf[(lane + 32 * r) * WF + c]);
                a = warp_minf(a);
            } else {
#pragma unroll
                for (int r = 1; r < UPD_THREADS / 32; r++) a = a + shf[(lane + 32 * r) * WF + c];
                a = warp_sumf(a);
            }
            if (lane == 0) partf[c] = a;
        }
        __syncthreads();
        if (t == 0) {
            const float a = partf[0], b = -partf[1];
            if (need_dt && a == a) {
                const double ad = (double)a;
                atomicMin(&st->newdt_bits, (unsigned long long)__double_as_longlong(ad));
            }
            if (b > 0) {
                const double bd = (double)b;
                atomicMax(&st->rmax_bits, (unsigned long long)__double_as_longlong(bd));
            }
            if (final_stage)
                for (int k = 0; k < 8; k++) A.red[8 * (size_t)blk + k] = (double)partf[2 + k];
        }
        return;
    } else if constexpr (!SPLIT) {
        // The smallest time step and the largest residual as integers (non-negative doubles
        // order as their bit patterns).  The eight sums, FP64, by halving: at each of the
        // first three exchanges a lane keeps half of its columns, so a warp adds 9 times
        // where a shuffle tree per column adds 40 (an FP64 instruction costs a warp 64
        // cycles with 1 lane active as with 32).  Fixed order.
        constexpr int NW = UPD_THREADS / 32;
        constexpr unsigned all = 0xffffffffu;
        __shared__ unsigned long long key[NW][2];
        __shared__ double shr[NW][8];
        if (need_dt) {
            const unsigned long long d = (unsigned long long)__double_as_longlong(dtc != dtc ? INFINITY : dtc);
            const unsigned h = __reduce_min_sync(all, (unsigned)(d >> 32));
            const unsigned l = __reduce_min_sync(all, (unsigned)(d >> 32) == h ? (unsigned)d : all);
            if (lane == 0) key[w][0] = ((unsigned long long)h << 32) | l;
        }
        const unsigned long long m = (unsigned long long)__double_as_longlong(rm);
        const unsigned h = __reduce_max_sync(all, (unsigned)(m >> 32));
        const unsigned l = __reduce_max_sync(all, (unsigned)(m >> 32) == h ? (unsigned)m : 0u);
        if (lane == 0) key[w][1] = ((unsigned long long)h << 32) | l;
        if (final_stage) {
            double v[8] = {ss[0], ss[1], ss[2], ss[3], vs[0], vs[1], vs[2], vs[3]};
#pragma unroll
            for (int n = 4, o = 16; n > 0; n >>= 1, o >>= 1) {
                const bool up = lane & o;
#pragma unroll
                for (int k = 0; k < 4; k++)
                    if (k < n) {
                        const double keep = up ? v[n + k] : v[k], give = up ? v[k] : v[n + k];
                        v[k] = keep + __shfl_xor_sync(all, give, o);
                    }
            }
            v[0] = v[0] + __shfl_xor_sync(all, v[0], 2);
            v[0] = v[0] + __shfl_xor_sync(all, v[0], 1);
            if ((lane & 3) == 0) shr[w][lane >> 2] = v[0];  // column: the kept halves' bits
        }
        __syncthreads();
        if (w != 0) return;
        if (final_stage) {
            const int c = lane & 7, g = lane >> 3;
            double v = shr[g][c];
            for (int k = g + 4; k < NW; k += 4) v = v + shr[k][c];
            v = v + __shfl_xor_sync(all, v, 8);
            v = v + __shfl_xor_sync(all, v, 16);
            if (lane < 8) A.red[8 * (size_t)blk + c] = v;
        }
        if (lane < 2 && (lane == 1 || need_dt)) {
            unsigned long long x = key[0][lane];
            for (int k = 1; k < NW; k++) x = lane ? max(x, key[k][1]) : min(x, key[k][0]);
            if (lane == 0)
                atomicMin(&st->newdt_bits, x);
            else if (x != 0ull)
                atomicMax(&st->rmax_bits, x);
        }
    }
}

inline int ret(cudaError_t e) { return e == cudaSuccess ? 0 : (int)e; }

template <typename T, int PR>
int launch_cell_pr(const DMesh &M, const DPhys &P, const DArrays &A, const T *qin, int limit, void *stream)
{
    const int TB = cell_threads<T, PR>();
    dim3 grid((M.C + TB - 1) / TB);
    if (grid.x == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    const bool lp = P.lp && P.limited;
    cudaError_t e;
    if constexpr (!is_fp32<T>) {
        // four threads per cell wherever k_cell4 holds: every mesh size is faster with it
        if (!lp && P.order > 1 && (M.soft || !is_fp64<T>)) {
            const int T4 = cell4_threads<T>();
            const dim3 g4((unsigned)((4 * (int64_t)M.C + T4 - 1) / T4)), b4(T4);
            if (M.maxJ <= 3)
                e = M.uniform ? launch_dep(k_cell4<T, 3, true>, g4, b4, s, M, P, A, qin, limit)
                              : launch_dep(k_cell4<T, 3, false>, g4, b4, s, M, P, A, qin, limit);
            else if (M.maxJ == 4)
                e = M.uniform ? launch_dep(k_cell4<T, 4, true>, g4, b4, s, M, P, A, qin, limit)
                              : launch_dep(k_cell4<T, 4, false>, g4, b4, s, M, P, A, qin, limit);
            else
                e = launch_dep(k_cell4<T, 6, false>, g4, b4, s, M, P, A, qin, limit);
            return ret(e);
        }
    }
#define EBB_CELL_U(MJ, U)                                                                 \
    if (lp)                                                                               \
        e = launch_dep(k_cell<T, MJ, true, U, PR>, grid, dim3(TB), s, M, P, A, qin, limit); \
    else                                                                                  \
        e = launch_dep(k_cell<T, MJ, false, U, PR>, grid, dim3(TB), s, M, P, A, qin, limit);
#define EBB_CELL(MJ)           \
    if (M.uniform) {           \
        EBB_CELL_U(MJ, true)   \
    } else {                   \
        EBB_CELL_U(MJ, false)  \
    }
    if (M.maxJ <= 3) {
        EBB_CELL(3)
    } else if (M.maxJ == 4) {
        EBB_CELL(4)
    } else {  // meshes of hexagons only are not specialised
        EBB_CELL_U(6, false)
    }
#undef EBB_CELL
#undef EBB_CELL_U
    return ret(e);
}

template <typename T, int PR>
int launch_flux_pr(const DMesh &M, const DPhys &P, const DArrays &A, const T *qin, void *stream)
{
    const int TB = flux_threads<T, PR>();
    int nbi = (M.Eint + TB - 1) / TB, nbb = (M.G + TB - 1) / TB;
    if (nbi + nbb == 0) return 0;
    return ret(launch_dep(k_flux<T, PR>, dim3(nbi + nbb), dim3(TB), (cudaStream_t)stream, M, P, A, qin, nbb));
}

template <typename T, int PR>
int launch_update_pr(const DMesh &M, const DPhys &P, const DArrays &A, int stage, const T *qin, T *qout,
                     int dt_update, int need_dt, int final_stage, void *stream)
{
    dim3 grid(M.n_upd_blocks);
    if (grid.x == 0) return 0;
    cudaStream_t s = (cudaStream_t)stream;
    cudaError_t e = cudaSuccess;
#define EBB_UPD_U(S, MJ, U)                                                                                        \
    e = launch_dep(k_update<T, S, MJ, U, PR>, grid, dim3(UPD_THREADS), s, M, P, A, qin, qout, dt_update, need_dt,   \
                   final_stage)
#define EBB_UPD(S)                                                                                                 \
    case S:                                                                                                        \
        if constexpr (PR == 2) { /* uniform meshes only */                                                         \
            if (M.maxJ <= 3)                                                                                       \
                EBB_UPD_U(S, 3, true);                                                                             \
            else                                                                                                   \
                EBB_UPD_U(S, 4, true);                                                                             \
        } else if (M.maxJ <= 3) {                                                                                  \
            if (M.uniform)                                                                                         \
                EBB_UPD_U(S, 3, true);                                                                             \
            else                                                                                                   \
                EBB_UPD_U(S, 3, false);                                                                            \
        } else if (M.maxJ == 4) {                                                                                  \
            if (M.uniform)                                                                                         \
                EBB_UPD_U(S, 4, true);                                                                             \
            else                                                                                                   \
                EBB_UPD_U(S, 4, false);                                                                            \
        } else {                                                                                                   \
            EBB_UPD_U(S, 6, false);                                                                                \
        }                                                                                                          \
        break;
    switch (stage) {
        EBB_UPD(ST_RESID)
        EBB_UPD(ST_EULER)
        EBB_UPD(ST_RK2_1)
        EBB_UPD(ST_RK2_2)
        EBB_UPD(ST_TVD_1)
        EBB_UPD(ST_TVD_2)
        EBB_UPD(ST_RK4_1)
        EBB_UPD(ST_RK4_2)
        EBB_UPD(ST_RK4_3)
        EBB_UPD(ST_RK4_4)
    default:
        return -1;
    }
#undef EBB_UPD
#undef EBB_UPD_U
    return ret(e);
}

// The launch-shape profile: split solves of inviscid meshes take their own shapes, large ones
// the second of two.  Up to the line a stage's data passes through L2 more than once: the cell
// kernel marks its geometry to leave it first, and the update kernel has all its loads in
// flight, at 48 registers and 40 warps per SM.  Beyond it both kernels run at the memory's
// rate, where evict-first loads and fewer warps lose: plain loads, and on uniform meshes an
// update kernel that loads each value where it is used, at 32 registers and 64 warps (mixed
// meshes spill there: 135 against 129 us a launch on 4M cells).  us a step, profile 1 / 2:
// triangles (RK2) 1M 159 / 163, 2M 294 / 296, 3M 435 / 426, 6M 840 / 827; quads (TVD-RK2) 1M
// 207.2 / 207.7, 4M 754 / 719, 16M 2928 / 2747; 512 bump channels, 24.3M triangles (TVD-RK2),
// 3672 / 3508.
constexpr int kLargeCells = 2500000;
template <typename T> int shape_profile(const DMesh &M, const DPhys &P)
{
    return !is_fp32<T> || P.viscous ? 0 : (M.C < kLargeCells ? 1 : 2);
}

template <typename T>
int launch_cell_impl(const DMesh &M, const DPhys &P, const DArrays &A, const T *qin, int limit, void *stream)
{
    if constexpr (is_fp32<T>) {
        const int p = shape_profile<T>(M, P);
        if (p == 1) return launch_cell_pr<T, 1>(M, P, A, qin, limit, stream);
        if (p == 2) return launch_cell_pr<T, 2>(M, P, A, qin, limit, stream);
    }
    return launch_cell_pr<T, 0>(M, P, A, qin, limit, stream);
}
template <typename T> int launch_flux_impl(const DMesh &M, const DPhys &P, const DArrays &A, const T *qin, void *stream)
{
    if constexpr (is_fp32<T>)
        if (shape_profile<T>(M, P)) return launch_flux_pr<T, 1>(M, P, A, qin, stream);
    return launch_flux_pr<T, 0>(M, P, A, qin, stream);
}
template <typename T>
int launch_update_impl(const DMesh &M, const DPhys &P, const DArrays &A, int stage, const T *qin, T *qout,
                       int dt_update, int need_dt, int final_stage, void *stream)
{
    if constexpr (is_fp32<T>) {
        const int p = shape_profile<T>(M, P);
        if (p == 2 && M.uniform && M.maxJ <= 4)
            return launch_update_pr<T, 2>(M, P, A, stage, qin, qout, dt_update, need_dt, final_stage, stream);
        if (p) return launch_update_pr<T, 1>(M, P, A, stage, qin, qout, dt_update, need_dt, final_stage, stream);
    }
    return launch_update_pr<T, 0>(M, P, A, stage, qin, qout, dt_update, need_dt, final_stage, stream);
}

// ---- ebb-reconstruct (app/reconstruct.d:239-424) --------------------------------
// Edge values 0.5 (q[0] + q[1]) of every edge, at its reference edge id.  q[1] of a
// boundary edge is what the boundary flux code of solve.d:769-968 leaves there:
// the exact state at the midpoint (Dirichlet), the freestream (fullState), the ghost
// state (inviscid wall, constant pressure, TP inflow), the face state with negated
// momentum (viscous wall) or with reflected velocity (symmetry).
template <typename T>
__global__ void k_recon_edges(DMesh M, DArrays A, const T *__restrict__ qs, double *out)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= M.Eint + M.G) return;
    const T *face = reinterpret_cast<const T *>(A.face);
    T q0[4], q1[4];
    int ref;
    if (e < M.Eint) {
        const int2 sl = reinterpret_cast<const int2 *>(M.e_slot)[e];
        ld4(face + 4 * (size_t)sl.x, q0);
        ld4(face + 4 * (size_t)sl.y, q1);
        ref = M.e_ref[e];
    } else {
        const int b = e - M.Eint;
        ld4(face + 4 * (size_t)M.b_slot[b], q0);
        ref = M.b_ref[b];
        const int type = M.b_type[b];
        switch (type & 0xff) {
        case BC_DIRICHLET:
            ld4(ptr<T>(M.g.b_dmid) + 4 * (size_t)b, q1);
            break;
        case BC_FULLSTATE:
            ld4(ptr<T>(M.g.b_data) + 4 * (size_t)b, q1);
            break;
        case BC_VISCWALL:
            q1[0] = q0[0];
            q1[1] = -q0[1];
            q1[2] = -q0[2];
            q1[3] = q0[3];
            break;
        case BC_SYMMETRY: {
            T v0 = q0[1] / q0[0], v1 = q0[2] / q0[0], n0, n1;
            reflect(type, ptr<T>(M.g.b_refl) + 4 * (size_t)b, v0, v1, n0, n1);
            q1[0] = q0[0];
            q1[1] = q0[0] * n0;
            q1[2] = q0[0] * n1;
            q1[3] = q0[3];
            break;
        }
        default:  // inviscid wall, constant pressure, TP inflow: the ghost state
            ld4(qs + 4 * ((size_t)M.C + b), q1);
        }
    }
#pragma unroll
    for (int k = 0; k < 4; k++) out[4 * (size_t)ref + k] = 0.5 * ((double)q0[k] + (double)q1[k]);
}

// Node values of the nodes the elements use.  Interior node: the average over the
// node's cells (reference element order) of q + lim0 g0 dx + lim1 g1 dy at the node
// (reconstruct.d:303-324); boundary node: the average of the edge values of the
// boundary edges its cells share with it (reconstruct.d:326-346).  A NaN value records
// the lowest node index in *err (reconstruct.d enforces no NaN).
template <typename T>
__global__ void k_recon_nodes(DMesh M, DArrays A, int n, const int32_t *__restrict__ off,
                              const int32_t *__restrict__ items, const uint8_t *__restrict__ is_b,
                              const double *__restrict__ nxy, const double *__restrict__ cxy,
                              const double *__restrict__ edge_vals, double *out, unsigned long long *err)
{
    const int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    double s[4] = {0.0, 0.0, 0.0, 0.0};
    const int a0 = off[v], a1 = off[v + 1];
    if (!is_b[v]) {
        const T *g = reinterpret_cast<const T *>(A.grad);
        const T *l = reinterpret_cast<const T *>(A.lim);
        for (int a = a0; a < a1; a++) {
            const int c = items[a];  // device cell
            const double dx = nxy[2 * (size_t)v] - cxy[2 * (size_t)c];
            const double dy = nxy[2 * (size_t)v + 1] - cxy[2 * (size_t)c + 1];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const double q = A.q64[4 * (size_t)c + k];
                const double g0 = (double)g[8 * (size_t)c + 2 * k], g1 = (double)g[8 * (size_t)c + 2 * k + 1];
                const double l0 = (double)l[8 * (size_t)c + 2 * k], l1 = (double)l[8 * (size_t)c + 2 * k + 1];
                s[k] += q + l0 * g0 * dx + l1 * g1 * dy;
            }
        }
    } else {
        for (int a = a0; a < a1; a++) {
            const int e = items[a];  // reference edge id
#pragma unroll
            for (int k = 0; k < 4; k++) s[k] += edge_vals[4 * (size_t)e + k];
        }
    }
    const double r = 1.0 / (double)(a1 - a0);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        s[k] *= r;
        out[4 * (size_t)v + k] = s[k];
    }
    if (isnan(s[0]) || isnan(s[1]) || isnan(s[2]) || isnan(s[3])) atomicMin(err, (unsigned long long)v);
}

template <typename T>
int launch_recon_impl(const DMesh &M, const DArrays &A, const T *qs, double *edge_out, int n_nodes,
                      const int32_t *off, const int32_t *items, const uint8_t *is_b, const double *nxy,
                      const double *cxy, double *node_out, unsigned long long *err, void *stream)
{
    cudaStream_t st = (cudaStream_t)stream;
    const int ne = M.Eint + M.G;
    if (ne > 0) k_recon_edges<T><<<(ne + 255) / 256, 256, 0, st>>>(M, A, qs, edge_out);
    if (n_nodes > 0)
        k_recon_nodes<T><<<(n_nodes + 255) / 256, 256, 0, st>>>(M, A, n_nodes, off, items, is_b, nxy, cxy, edge_out,
                                                                node_out, err);
    return ret(cudaGetLastError());
}

}  // namespace ebbdev

#define EBB_INSTANTIATE(T)                                                                                        \
    template <>                                                                                                   \
    int launch_cell<T>(const DMesh &M, const DPhys &P, const DArrays &A, const T *qin, int limit, void *stream)  \
    {                                                                                                             \
        return ebbdev::launch_cell_impl<T>(M, P, A, qin, limit, stream);                                          \
    }                                                                                                             \
    template <>                                                                                                   \
    int launch_flux<T>(const DMesh &M, const DPhys &P, const DArrays &A, const T *qin, void *stream)              \
    {                                                                                                             \
        return ebbdev::launch_flux_impl<T>(M, P, A, qin, stream);                                                 \
    }                                                                                                             \
    template <>                                                                                                   \
    int launch_update<T>(const DMesh &M, const DPhys &P, const DArrays &A, int stage, const T *qin, T *qout,      \
                         int dt_update, int need_dt, int final_stage, void *stream)                               \
    {                                                                                                             \
        return ebbdev::launch_update_impl<T>(M, P, A, stage, qin, qout, dt_update, need_dt, final_stage, stream); \
    }                                                                                                             \
    template <>                                                                                                   \
    int launch_recon<T>(const DMesh &M, const DArrays &A, const T *qs, double *edge_out, int n_nodes,            \
                        const int32_t *off, const int32_t *items, const uint8_t *is_b, const double *nxy,         \
                        const double *cxy, double *node_out, unsigned long long *err, void *stream)               \
    {                                                                                                             \
        return ebbdev::launch_recon_impl<T>(M, A, qs, edge_out, n_nodes, off, items, is_b, nxy, cxy, node_out,   \
                                            err, stream);                                                         \
    }
