// k_fp64.cu -- plain FP64 instantiation of the stage kernels, plus the time-loop
// epilogue, the flux seam and the state copy kernels (sm_103a).
//
// Compiled with -fmad=false: every multiply and add rounds separately, in the
// reference's left-to-right order, so results are bitwise those of the FP64 CPU
// path (up to the sign of exact zeros) except where CUDA's pow() is used
// (constant-pressure ghost states).
#include "../../include/ebb_gb300.h"
#include "kernels.cuh"

EBB_INSTANTIATE(double)

using namespace ebbdev;

namespace {

// end of one runIntegrator iteration (app/solver.d:126-249).  blockIdx.x: the instance (an
// arena may have more than the 65,535 that the grid's other dimensions hold); blockIdx.y: a
// part of its rows of block partial sums (step_parts of them, a function of the instance's
// size alone, so that an instance sums in the same order in any arena).
// The block that finishes last adds the parts up in order and runs the epilogue.
//
// What bounds it is latency: an FP64 addition takes a warp 64 cycles, so a thread here
// holds one column of the eight (one addition per row, 32 rows apart), and the epilogue's
// square roots, quotients and products sit in different lanes.  Against one block per
// instance with all ten columns per thread and a serial epilogue: 40 instances of up to
// 60,000 cells 13.2 -> 8.6 us; steps of 6,000 cells 29.8 -> 23.7 us, of 500,000 (two
// stages) 101 -> 91 us, of 1M (four stages, 16 parts) 466 -> 450 us, all split precision.
template <typename T> __global__ void __launch_bounds__(EBB_RED_THREADS) k_step_end(DMesh M, DArrays A, int nblk)
{
    const int inst = blockIdx.x, part = blockIdx.y;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    DState *st = A.st + inst;
    const int b0 = M.inst_blk ? M.inst_blk[inst] : 0, b1 = M.inst_blk ? M.inst_blk[inst + 1] : nblk;
    const int fb0 = M.force_off ? M.force_off[inst] : 0, fb1 = M.force_off ? M.force_off[inst + 1] : M.n_force;
    const int ncell = M.inst_c0 ? M.inst_c0[inst + 1] - M.inst_c0[inst] : M.C;
    const int parts = step_parts(b1 - b0);
    grid_dep_release();
    grid_dep_wait();
    if (part >= parts || st->done) return;
    if (st->err_key != EBB_NOERR) {
        if (part == 0 && t == 0) st->done = 1;
        return;
    }
    __shared__ double sh[EBB_RED_THREADS / 32][10];
    __shared__ int last;
    // column t % 8 of rows t / 8, t / 8 + 32, ... of this part
    const int rows = (b1 - b0 + parts - 1) / parts, r0 = b0 + part * rows, r1 = min(r0 + rows, b1);
    double s = 0.0, f0 = 0.0, f1 = 0.0;
#pragma unroll 4
    for (int r = r0 + (t >> 3); r < r1; r += EBB_RED_THREADS / 8) s = s + A.red[8 * (size_t)r + (t & 7)];
    const T *fl = reinterpret_cast<const T *>(A.fl);
    for (int f = fb0 + part * EBB_RED_THREADS + t; f < fb1; f += parts * EBB_RED_THREADS) {
        const size_t e = (size_t)M.Eint + M.force_b[f];
        f0 = f0 + (double)fl[4 * e + 1];
        f1 = f1 + (double)fl[4 * e + 2];
    }
    s = s + __shfl_down_sync(0xffffffffu, s, 16);
    s = s + __shfl_down_sync(0xffffffffu, s, 8);
    if (lane < 8) sh[w][lane] = s;
    if (fb1 > fb0) {
        f0 = warp_sum(f0);
        f1 = warp_sum(f1);
    }
    if (lane == 0) {
        sh[w][8] = f0;
        sh[w][9] = f1;
    }
    __syncthreads();
    if (w != 0) return;
    double v = 0.0;  // lane c < 10: the sum of column c
    if (lane < 10)
        for (int k = 0; k < EBB_RED_THREADS / 32; k++) v = k ? v + sh[k][lane] : sh[0][lane];
    if (parts > 1) {
        double *p = A.endp + 10 * EBB_STEP_PARTS * (size_t)inst;
        if (lane < 10) p[10 * part + lane] = v;
        __threadfence();
        __syncwarp();
        if (lane == 0) last = atomicAdd(&st->end_count, 1u) == (unsigned)parts - 1u;
        __syncwarp();
        if (!last) return;
        __threadfence();
        if (lane < 10) {
            const volatile double *q = p;
            v = q[lane];
            for (int k = 1; k < parts; k++) v = v + q[10 * k + lane];
        }
    }
    const unsigned all = 0xffffffffu;
    // lanes 0-3: the residual of each component; 4, 5: drag and lift; 6: dt / 6; 7: t + dt
    const double vs = __shfl_sync(all, v, (lane & 3) + 4), fx = __shfl_sync(all, v, 8), fy = __shfl_sync(all, v, 9);
    const double dt = st->dynamic_dt ? __longlong_as_double((long long)st->newdt_bits) : st->dt;
    double x = 0.0;
    if (lane < 4)
        x = ratio(root((double)ncell * v), vs);
    else if (lane < 6)
        x = st->rot[2 * (lane - 4)] * fx + st->rot[2 * (lane - 4) + 1] * fy;
    else if (lane == 6)
        x = ratio(dt, 6.0);
    else if (lane == 7)
        x = st->t + dt;
    double resid[4];
#pragma unroll
    for (int k = 0; k < 4; k++) resid[k] = __shfl_sync(all, x, k);
    const double drag = __shfl_sync(all, x, 4), lift = __shfl_sync(all, x, 5), sixth = __shfl_sync(all, x, 6),
                 tnext = __shfl_sync(all, x, 7);
    if (lane != 0) return;
    const double rmax = __longlong_as_double((long long)st->rmax_bits);
    const double residMax = fmax(fmax(resid[0], resid[1]), fmax(resid[2], resid[3]));
    if (st->cfl_adjust) {
        if (st->resid_last < residMax)
            st->resid_inc++;
        else if (st->resid_inc >= 1)
            st->resid_inc--;
        if (st->resid_inc >= 2000) {
            st->cfl *= 0.99;
            st->cflf = (float)st->cfl;
            st->resid_inc = 0;
        }
    }
    st->resid_last = residMax;
    if (st->resid_first < 0) st->resid_first = resid[0];
    if (resid[0] < st->resid_min) {
        st->resid_min = resid[0];
        st->resid_min_iter = st->iter;
    }
    st->last[0] = drag;
    st->last[1] = lift;
#pragma unroll
    for (int k = 0; k < 4; k++) st->last[2 + k] = resid[k];
    st->last[6] = rmax;
    if (st->rec_enabled) {
        DRecord &r = A.rec[st->n_rec % EBB_REC_CAP];
        r.t = st->t;
        r.drag = drag;
        r.lift = lift;
#pragma unroll
        for (int k = 0; k < 4; k++) r.resid[k] = resid[k];
        r.rmax = rmax;
        r.dt = dt;
        r.cfl = st->cfl;
        st->n_rec++;
    }
    st->t = tnext;
    st->iter++;
    st->done = !(st->t < st->t_end) || (st->max_steps > 0 && st->iter >= st->max_steps) ||
               (st->stop_drop > 0 && resid[0] <= st->stop_drop * st->resid_first) ||
               (st->stall_steps > 0 && st->resid_min <= 1e-3 * st->resid_first &&
                st->iter - st->resid_min_iter > st->stall_steps);
    set_step(*st, dt, 0.5 * dt, sixth);
    st->newdt_bits = 0x7FF0000000000000ull;  // +inf
    st->rmax_bits = 0ull;
    st->end_count = 0u;
}

__global__ void k_flux_batch(int kind, int64_t n, const double *qL, const double *qR, const double *nrm, double *F,
                             double *s)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double a[4], b[4], f[4], sm;
    ld4(qL + 4 * i, a);
    ld4(qR + 4 * i, b);
    inviscid_flux(kind, a, b, nrm[2 * i], nrm[2 * i + 1], f, sm);
    st4(F + 4 * i, f);
    s[i] = sm;
}

// gather: dst[i] = src[idx[i]]; scatter: dst[idx[i]] = src[i]  (4 doubles per item)
__global__ void k_permute4(const double *__restrict__ src, double *__restrict__ dst, const int32_t *__restrict__ idx,
                           int64_t n, int gather)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v[4];
    if (gather) {
        ld4(src + 4 * (size_t)idx[i], v);
        st4(dst + 4 * (size_t)i, v);
    } else {
        ld4(src + 4 * (size_t)i, v);
        st4(dst + 4 * (size_t)idx[i], v);
    }
}

__global__ void k_to_float4(const double *__restrict__ src, float *__restrict__ dst, int64_t n)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v[4];
    ld4(src + 4 * i, v);
    float f[4] = {(float)v[0], (float)v[1], (float)v[2], (float)v[3]};
    st4(dst + 4 * i, f);
}

__global__ void k_to_double4(const float *__restrict__ src, double *__restrict__ dst, int64_t n)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float f[4];
    ld4(src + 4 * i, f);
    double v[4] = {(double)f[0], (double)f[1], (double)f[2], (double)f[3]};
    st4(dst + 4 * i, v);
}

// State in and out in the caller's cell order.  The reference-order side is read or
// written in sequence (the device side through the inverse permutation), so when it
// is a page-locked host buffer the link carries whole contiguous lines.
__global__ void k_load_state(const double *__restrict__ src, double *__restrict__ q64, float *__restrict__ qs1,
                             const int32_t *__restrict__ iperm, int64_t n)
{
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double v[4];
    ld4(src + 4 * j, v);
    const size_t i = (size_t)iperm[j];
    st4(q64 + 4 * i, v);
    if (qs1) {
        float f[4] = {(float)v[0], (float)v[1], (float)v[2], (float)v[3]};
        st4(qs1 + 4 * i, f);
    }
}

__global__ void k_store_state(const double *__restrict__ q64, double *__restrict__ dst,
                              const int32_t *__restrict__ iperm, int64_t n)
{
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    double v[4];
    ld4(q64 + 4 * (size_t)iperm[j], v);
    st4(dst + 4 * j, v);
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

int update_blocks(int C) { return (C + UPD_THREADS - 1) / UPD_THREADS; }

int update_grid(const DMesh &M) { return M.n_upd_blocks; }

int launch_step_end(const DMesh &M, const DArrays &A, int nred_blocks, int precision, void *stream)
{
    const int n = M.n_inst > 0 ? M.n_inst : 1;
    const dim3 grid(n, step_parts(M.max_inst_blocks)), block(EBB_RED_THREADS);
    const cudaStream_t q = (cudaStream_t)stream;
    cudaError_t e;
    if (precision == EBB_PREC_SPLIT)
        e = launch_dep(k_step_end<float>, grid, block, q, M, A, nred_blocks);
    else if (precision == EBB_PREC_DF)
        e = launch_dep(k_step_end<ebbdf::df>, grid, block, q, M, A, nred_blocks);
    else
        e = launch_dep(k_step_end<double>, grid, block, q, M, A, nred_blocks);
    return ret(e);
}

int launch_flux_batch(int kind, int64_t n, const double *qL, const double *qR, const double *nrm, double *F, double *s,
                      void *stream)
{
    if (n <= 0) return 0;
    k_flux_batch<<<nblk(n, 128), 128, 0, (cudaStream_t)stream>>>(kind, n, qL, qR, nrm, F, s);
    return ret(cudaGetLastError());
}

int launch_permute4(const double *src, double *dst, const int32_t *idx, int64_t n, int gather, void *stream)
{
    if (n <= 0) return 0;
    k_permute4<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(src, dst, idx, n, gather);
    return ret(cudaGetLastError());
}

int launch_to_float4(const double *src, float *dst, int64_t n, void *stream)
{
    if (n <= 0) return 0;
    k_to_float4<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(src, dst, n);
    return ret(cudaGetLastError());
}

int launch_to_double4(const float *src, double *dst, int64_t n, void *stream)
{
    if (n <= 0) return 0;
    k_to_double4<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(src, dst, n);
    return ret(cudaGetLastError());
}

int launch_load_state(const double *src, double *q64, float *qs1, const int32_t *iperm, int64_t n, void *stream)
{
    if (n <= 0) return 0;
    k_load_state<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(src, q64, qs1, iperm, n);
    return ret(cudaGetLastError());
}

int launch_store_state(const double *q64, double *dst, const int32_t *iperm, int64_t n, void *stream)
{
    if (n <= 0) return 0;
    k_store_state<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(q64, dst, iperm, n);
    return ret(cudaGetLastError());
}
