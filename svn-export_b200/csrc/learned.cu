// Flexible CG, the Chebyshev-Jacobi polynomial preconditioner (the fallback of the learned
// method) and the training pairs of the plain solver.  No counterpart in the reference, which
// solves with PETSc's CG and ILU (src/la/solve.cc:370).
#include <cuda_runtime.h>

#include "device_system.hpp"
#include "learned.hpp"
#include "pdl.hpp"

namespace mh {

namespace {

struct Plan {
    const int32_t *inst, *tile_begin, *tile_end, *inst_blk;
};

Plan plan32(const DevSystem &s) {
    const DevPlan &p = s.plan[1];
    return {p.blk_inst, p.tile_begin, p.tile_end, p.inst_blk};
}

template <int NV> struct Sums { double v[NV]; };

template <int NV> __device__ __forceinline__ Sums<NV> block_sum(Sums<NV> s) {
    __shared__ double sh[kWarpsPerBlock][NV];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        double v = s.v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) sh[warp][k] = v;
    }
    __syncthreads();
    Sums<NV> out;
#pragma unroll
    for (int k = 0; k < NV; ++k) out.v[k] = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < kWarpsPerBlock; ++w)
#pragma unroll
            for (int k = 0; k < NV; ++k) out.v[k] += sh[w][k];
    __syncthreads();
    return out;
}

// Same contract as the Krylov kernels' block_finish (solver.cu): publish the block partial,
// the instance's last-arriving block gets the totals (thread 0).
template <int NV>
__device__ __forceinline__ bool block_finish(Sums<NV> s, double *partial, InstCtl *c, const Plan &plan, int inst,
                                             Sums<NV> &tot) {
    __shared__ bool am_last;
    Sums<NV> b = block_sum<NV>(s);
    const int pb = plan.inst_blk[inst], pe = plan.inst_blk[inst + 1];
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < NV; ++k) partial[(int64_t)blockIdx.x * 4 + k] = b.v[k];
        __threadfence();
        am_last = (atomicAdd(&c->ticket, 1u) == (unsigned)(pe - pb) - 1);
    }
    __syncthreads();
    if (!am_last) return false;
    __threadfence();
    Sums<NV> a;
#pragma unroll
    for (int k = 0; k < NV; ++k) a.v[k] = 0.0;
    for (int t = pb + threadIdx.x; t < pe; t += blockDim.x)
#pragma unroll
        for (int k = 0; k < NV; ++k) a.v[k] += __ldcg(&partial[(int64_t)t * 4 + k]);
    tot = block_sum<NV>(a);
    if (threadIdx.x == 0) c->ticket = 0u;
    return true;
}

__device__ __forceinline__ void finish_inst(InstCtl *c, int status, int32_t *n_done) {
    c->done = 1;
    c->status = status;
    atomicAdd(n_done, 1);
}

// (S^ v)[row]
__device__ __forceinline__ float sell_row_dot(const SellView<float> &A, const float *__restrict__ v, int64_t sl,
                                              int lane) {
    const int64_t off = A.slice_off[sl];
    const int w = (int)((A.slice_off[sl + 1] - off) / kSliceRows);
    float acc = 0.f;
    for (int j = 0; j < w; ++j) {
        const int64_t slot = off + (int64_t)j * kSliceRows + lane;
        acc += __ldcs(A.val + slot) * v[__ldcs(A.col + slot)];
    }
    return acc;
}

// ---- flexible CG ------------------------------------------------------------------------
// One iteration after z = M r is two kernels (beta, the direction, S^ p and the update as kernels of
// their own were four, and each ends in a last-block reduction that the next one waits for):
//   k_fcg_spmv:   s = S^ z with the sums z.q, z.r, p.r, z.s over the previous direction (p, q = S^ p);
//                 the last block forms beta = z.q / p.q, the new direction's p.r = z.r - beta p.r and
//                 p.q = z.s - beta z.q (S^ is symmetric and z.S^ p = z.q), alpha = p.r / p.q;
//   k_fcg_update: p = z - beta p, q = s - beta q, x += alpha p, r -= alpha q, r.r, stopping test.
// q follows the direction's recurrence instead of a product with the new p, so what p, q and s are
// rounded to stays in q for the rest of the run: the three are FP64 (z, x and r are FP32).
// Residual after one segment of 800 iterations (158k rows, recursion at 1.2e-8): 6.0e-8 with q a product of
// FP32 vectors, 7.4e-8 with the recurrence in FP32, 5.9e-8 in FP64.  The row entries go two to a load in the
// update; z and r are loaded a tile ahead with the slots in the product, p and q beside the gathers.
// The blocks of an instance take its tiles in turn (solver.cu, Tiles).
// Measured (B200, us an iteration without the preconditioner, four kernels over neighbouring tiles
// -> two with all vectors FP32): 52k rows 20 -> 11, 3.2M 96 -> 68, 10.9M 381 -> 233.  The FP64 ones are 32
// bytes a row more; a multigrid iteration with them, against all FP32: 67.0 us and 66.7 (52k edges), 119.4 and
// 118.4 (405k), 251 and 246 (1.35M), 471 and 458 (3.2M), 2075 and 2019 (11M).
struct FcgStage {
    static constexpr int kJ = 6;
    int64_t off;
    int w;
    int32_t c[kJ];
    float v[kJ];
    float dg, z, r;
};

__device__ __forceinline__ void fcg_stage_load(const SellView<float> &A, int tile, FcgStage &st) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t sl = (int64_t)tile * kWarpsPerBlock + warp;
    st.off = A.slice_off[sl];
    st.w = (int)((A.slice_off[sl + 1] - st.off) / kSliceRows);
    st.dg = __ldcs(A.val + st.off + lane);  // a row's first slot is its diagonal
#pragma unroll
    for (int j = 0; j < FcgStage::kJ; ++j) {
        const bool in = j + 1 < st.w;
        const int64_t slot = st.off + (int64_t)(j + 1) * kSliceRows + lane;
        st.c[j] = in ? __ldcs(A.col + slot) : 0;
        st.v[j] = in ? __ldcs(A.val + slot) : 0.f;
    }
}
__device__ __forceinline__ void fcg_stage_load_vec(const float *z, const float *r, int tile, FcgStage &st) {
    const int64_t row = ((int64_t)tile * kWarpsPerBlock + (threadIdx.x >> 5)) * kSliceRows + (threadIdx.x & 31);
    st.z = z[row];
    st.r = r[row];
}

__global__ void __launch_bounds__(kBlockThreads, 4)
    k_fcg_spmv(SellView<float> A, const float *z, const float *r, const double *p, const double *q, double *s,
               double *partial, InstCtl *ctl, Plan plan, int32_t *n_done) {
    const int inst = plan.inst[blockIdx.x];
    InstCtl *c = ctl + inst;
    // the instance's blocks take its tiles in turn, so that all of them gather from one moving window
    const int pb = plan.inst_blk[inst], nb = plan.inst_blk[inst + 1] - pb;
    const int tb = plan.tile_begin[pb] + ((int)blockIdx.x - pb), te = plan.tile_end[pb + nb - 1];
    FcgStage st;
    if (tb < te) fcg_stage_load(A, tb, st);
    pdl_wait();
    if (c->done) return;
    const bool have = c->aux[1] != 0.0 && c->aux[0] != 0.0;  // else (p, q) may hold a broken direction
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    constexpr int kJ = FcgStage::kJ;
    Sums<4> t = {{0.0, 0.0, 0.0, 0.0}};
    if (tb < te) fcg_stage_load_vec(z, r, tb, st);
    for (int tile = tb; tile < te; tile += nb) {
        float g[kJ];
#pragma unroll
        for (int j = 0; j < kJ; ++j) g[j] = z[st.c[j]];
        const int64_t row = ((int64_t)tile * kWarpsPerBlock + warp) * kSliceRows + lane;
        const double pv = have ? p[row] : 0.0, qv = have ? q[row] : 0.0;
        const FcgStage cur = st;
        if (tile + nb < te) {
            fcg_stage_load(A, tile + nb, st);
            fcg_stage_load_vec(z, r, tile + nb, st);
        }
        double y = (double)cur.dg * (double)cur.z;
#pragma unroll
        for (int j = 0; j < kJ; ++j) y += (double)cur.v[j] * (double)g[j];
        for (int j = kJ + 1; j < cur.w; ++j) {
            const int64_t slot = cur.off + (int64_t)j * kSliceRows + lane;
            y += (double)__ldcs(A.val + slot) * (double)z[__ldcs(A.col + slot)];
        }
        s[row] = y;
        t.v[0] += (double)cur.z * qv;
        t.v[1] += (double)cur.z * (double)cur.r;
        t.v[2] += pv * (double)cur.r;
        t.v[3] += (double)cur.z * y;
    }
    Sums<4> tot;
    if (block_finish<4>(t, partial, c, plan, inst, tot) && threadIdx.x == 0) {
        const double beta = have ? tot.v[0] / c->aux[0] : 0.0;  // (p.q of the iteration before)
        const double pr = tot.v[1] - beta * tot.v[2], pq = tot.v[3] - beta * tot.v[0];
        c->rho = pr;
        c->beta = beta;
        c->alpha = 0.0;
        c->aux[2] = pq;
        if (!isfinite(pr)) finish_inst(c, -6, n_done);
        else if (pr == 0.0) finish_inst(c, 0, n_done);
        else if (!(pq > 0.0) || !isfinite(pq)) finish_inst(c, isfinite(pq) ? -8 : -6, n_done);
        else c->alpha = pr / pq;
    }
}

__global__ void __launch_bounds__(kBlockThreads)
    k_fcg_update(float2 *x, float2 *r, double2 *p, double2 *q, const float2 *z, const double2 *s, double *partial,
                 InstCtl *ctl, Plan plan, int32_t *n_done) {
    const int inst = plan.inst[blockIdx.x];
    InstCtl *c = ctl + inst;
    const int pb = plan.inst_blk[inst], nb = plan.inst_blk[inst + 1] - pb;
    const int t0 = plan.tile_begin[pb], t1 = plan.tile_end[pb + nb - 1];
    pdl_wait();
    if (c->done) return;
    const double alpha = c->alpha, beta = c->beta;
    double rr = 0.0;
    // beta = 0 starts a new direction sequence: p and q are not used (they may hold a broken one)
    auto dir = [&](double a, double b) { return beta == 0.0 ? a : a - beta * b; };
    auto one = [&](float zv, double sv, double &pv, double &qv, float &xv, float &rv) {
        pv = dir((double)zv, pv);
        qv = dir(sv, qv);
        xv = (float)((double)xv + alpha * pv);
        rv = (float)((double)rv - alpha * qv);
        rr += (double)rv * (double)rv;
    };
    // two rows a thread and turn: two tiles at a time of the instance's run, the blocks in turn
    constexpr int64_t kPer = kBlockThreads / 2;
    const int64_t i0 = t0 * kPer, end = t1 * kPer;
    for (int64_t i = i0 + ((int64_t)blockIdx.x - pb) * kBlockThreads + threadIdx.x; i < end;
         i += (int64_t)nb * kBlockThreads) {
        const float2 zv = __ldcs(z + i);
        const double2 sv = __ldcs(s + i);
        double2 pv = p[i], qv = q[i];
        float2 xv = x[i], rv = r[i];
        one(zv.x, sv.x, pv.x, qv.x, xv.x, rv.x);
        one(zv.y, sv.y, pv.y, qv.y, xv.y, rv.y);
        p[i] = pv;
        q[i] = qv;
        x[i] = xv;
        r[i] = rv;
    }
    Sums<1> t = {{rr}};
    Sums<1> tot;
    if (block_finish<1>(t, partial, c, plan, inst, tot) && threadIdx.x == 0) {
        c->aux[0] = c->aux[2];  // p.q of this iteration
        c->aux[1] = 1.0;        // (p, q) hold a direction the next one is made conjugate to
        c->rr = tot.v[0];
        c->iter += 1;
        if (!isfinite(tot.v[0])) finish_inst(c, -6, n_done);
        else if (tot.v[0] <= c->tol2) finish_inst(c, 0, n_done);
        else if (c->iter >= c->max_it) finish_inst(c, 1, n_done);
    }
}

// ---- Chebyshev-Jacobi polynomial preconditioner z = P_d(S^) r on [lo, hi] ---------------
// step 0: d = r / theta, z = d;  step k: d = c1 d + c2 (r - S^ z_prev), z = z_prev + d.
__global__ void __launch_bounds__(kBlockThreads)
    k_cheb_step(SellView<float> A, const float *r, const float *z_prev, float *z_next, float *d, double c1, double c2,
                int first, const InstCtl *ctl, Plan plan) {
    const int inst = plan.inst[blockIdx.x], tb = plan.tile_begin[blockIdx.x], te = plan.tile_end[blockIdx.x];
    pdl_wait();
    if (ctl[inst].done) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int tile = tb; tile < te; ++tile) {
        const int64_t sl = (int64_t)tile * kWarpsPerBlock + warp;
        const int64_t row = sl * kSliceRows + lane;
        float zn;
        if (first) {
            const float dn = (float)(c2 * (double)r[row]);
            d[row] = dn;
            zn = dn;
        } else {
            const double res = (double)r[row] - (double)sell_row_dot(A, z_prev, sl, lane);
            const float dn = (float)(c1 * (double)d[row] + c2 * res);
            d[row] = dn;
            zn = z_prev[row] + dn;
        }
        z_next[row] = zn;
    }
}

// Gershgorin bound max_i sum_j |S^_ij| (upper bound of the spectrum of S^)
__global__ void k_row_abs_max(SellView<float> A, int64_t n_rows, unsigned int *out) {
    const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    float s = 0.f;
    if (row < n_rows) {
        const int64_t sl = row / kSliceRows;
        const int lane = (int)(row % kSliceRows);
        const int64_t off = A.slice_off[sl];
        const int w = (int)((A.slice_off[sl + 1] - off) / kSliceRows);
        for (int j = 0; j < w; ++j) s += fabsf(A.val[off + (int64_t)j * kSliceRows + lane]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = fmaxf(s, __shfl_xor_sync(0xffffffffu, s, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, __float_as_uint(s));  // non-negative floats order as ints
}

// ---- training pairs of the plain solver --------------------------------------------
__global__ void k_pair_make(const double *__restrict__ xs, const double *__restrict__ x,
                            const double *__restrict__ r64, float *__restrict__ e, float *__restrict__ r, int64_t n,
                            double *acc) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    double rr = 0.0, er = 0.0;
    if (i < n) {
        const float ev = (float)(xs[i] - x[i]), rv = (float)r64[i];
        e[i] = ev;
        r[i] = rv;
        rr = (double)rv * (double)rv;
        er = (double)ev * (double)rv;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        rr += __shfl_xor_sync(0xffffffffu, rr, o);
        er += __shfl_xor_sync(0xffffffffu, er, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(acc, rr);
        atomicAdd(acc + 1, er);
    }
}

__global__ void k_pair_scale(float *__restrict__ e, float *__restrict__ r, float s, int64_t n) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        e[i] *= s;
        r[i] *= s;
    }
}

inline unsigned blocks_for(int64_t n, int th) { return (unsigned)((n + th - 1) / th); }

}  // namespace

cudaError_t launch_cheb_apply(const DevSystem &sys, const float *r, float *z0, float *z1, float *d, float *z_final,
                              int degree, double lo, double hi, cudaStream_t s, bool follows) {
    if (sys.rows_per_thread != 1) return cudaErrorInvalidValue;  // tiles of 256 rows
    const SellView<float> A = {sys.n_rows, sys.slice_off, sys.col, sys.val32};
    const unsigned g = (unsigned)sys.plan[1].n_blocks;
    const Plan p = plan32(sys);
    const double theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo), sigma = theta / delta;
    double rho = 1.0 / sigma;
    const float *zp = nullptr;
    for (int k = 0; k < degree; ++k) {
        double c1 = 0.0, c2 = 1.0 / theta;
        if (k > 0) {
            const double rho_new = 1.0 / (2.0 * sigma - rho);
            c1 = rho_new * rho;
            c2 = 2.0 * rho_new / delta;
            rho = rho_new;
        }
        const bool last = k == degree - 1;
        float *zn = last ? z_final : ((k % 2 == 0) ? z0 : z1);
        launch_chained(follows || k > 0, k_cheb_step, g, kBlockThreads, s, A, r, zp, zn, d, c1, c2, k == 0 ? 1 : 0,
                       sys.ctl, p);
        zp = zn;
    }
    return cudaGetLastError();
}

cudaError_t launch_fcg_iteration(const DevSystem &sys, const float *z, cudaStream_t s, bool chained) {
    if (sys.rows_per_thread != 1) return cudaErrorInvalidValue;  // tiles of 256 rows
    const SellView<float> A = {sys.n_rows, sys.slice_off, sys.col, sys.val32};
    const unsigned g = (unsigned)sys.plan[1].n_blocks;
    // (rows start on cudaMalloc's boundary)
    auto f2 = [](float *v) { return reinterpret_cast<float2 *>(v); };
    auto d2 = [](double *v) { return reinterpret_cast<double2 *>(v); };
    const cudaError_t e = launch_chained(chained, k_fcg_spmv, g, kBlockThreads, s, A, z, sys.r32, sys.p, sys.q, sys.s,
                                         sys.partial, sys.ctl, plan32(sys), sys.n_done);
    if (e != cudaSuccess) return e;
    return launch_chained(true, k_fcg_update, g, kBlockThreads, s, f2(sys.x32), f2(sys.r32), d2(sys.p), d2(sys.q),
                          reinterpret_cast<const float2 *>(z), d2(sys.s), sys.partial, sys.ctl, plan32(sys),
                          sys.n_done);
}

cudaError_t launch_spectrum_bound(const DevSystem &sys, unsigned int *out, cudaStream_t s) {
    const SellView<float> A = {sys.n_rows, sys.slice_off, sys.col, sys.val32};
    cudaError_t e = cudaMemsetAsync(out, 0, sizeof(unsigned int), s);
    if (e != cudaSuccess) return e;
    k_row_abs_max<<<blocks_for(sys.n_rows, 256), 256, 0, s>>>(A, sys.n_rows, out);
    return cudaGetLastError();
}

// (r, e) of one training pair: e = x* - x, r = the solver's residual (FP32), with |r|^2 and
// e.r summed into acc
cudaError_t launch_pair_make(int64_t n, const double *xs, const double *x, const double *r64, float *e, float *r,
                             double *acc, cudaStream_t s) {
    cudaError_t err = cudaMemsetAsync(acc, 0, 2 * sizeof(double), s);
    if (err != cudaSuccess) return err;
    k_pair_make<<<blocks_for(n, 256), 256, 0, s>>>(xs, x, r64, e, r, n, acc);
    return cudaGetLastError();
}

cudaError_t launch_pair_scale(int64_t n, float *e, float *r, float scale, cudaStream_t s) {
    k_pair_scale<<<blocks_for(n, 256), 256, 0, s>>>(e, r, scale, n);
    return cudaGetLastError();
}

}  // namespace mh
