// The Krylov run of a system that fits in the chip's shared memory: one cooperative launch whose
// blocks keep their rows of S^ and their part of the vectors on the SM for the whole run.  Same
// recurrences, FP64 sums and stopping test as the two-kernel iteration of solver.cu (KSPSolve on
// schur2, src/la/solve.cc:447-460).
//
// What bounds the two-kernel iteration at these sizes is latency: two launches of 5-6 us each
// (a gate, a block plan, slots, gathers, a last-block reduction) that move data worth well under
// 1 us.  Here an iteration has one grid-wide exchange:
//   A  q = S^ p for the block's rows, all from shared memory; partial sums p.q, r.q, q.q and the
//      r.r of the residual the iteration started from;
//   X  every q goes to L2 and every block publishes its four sums, each value in one atomic store
//      together with the exchange's number as its tag; the readers poll the values themselves, so
//      there is no counter, no fence and no second trip for the data.  Sums are added in block
//      order: the scalars are the same everywhere and deterministic;
//   B  r.r decides whether the run ended with the last update; else alpha, beta, and the update
//      of x, r, p.  The block also holds r and p of the rows its own rows couple to in other
//      blocks (the halo) and updates them with the owner's q, operation for operation as the
//      owner does, so p never has to be exchanged and a second grid barrier is not needed.
// q and the sums have two buffers: a block can be at most one exchange ahead of another.
// Rows are cut into contiguous runs of 32-row slices, balanced by bytes; columns are 16-bit
// indices into the block's own and halo entries, the diagonal is kept apart.
// The launch is cooperative, so all blocks are on the chip together; every poll is bounded, and a
// block that gives up sets *err and leaves: the vectors and the exchange buffers are then worth
// nothing, and the host starts the run again with the two-kernel iteration.
// The smallest systems run in one thread-block cluster instead (k_cg_cluster below).
// Measured (B200, us an iteration, two-kernel iteration -> this one): FP64, 6.9k edges 10.8 -> 2.8,
// 52k 11.7 -> 3.1, 175k 15.5 -> 4.6, 273k 17.7 -> 5.3; FP32, 52k 12.8 -> 3.5, 244k 17.1 -> 4.8,
// 528k 21.0 -> 7.5.  What is left is the exchange, about 2.2 us (two trips through L2, three block
// barriers), and from 200k edges on the FP64 arithmetic and conversions on the rows of one SM.
#include <algorithm>

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include "device_system.hpp"
#include "resident.hpp"

namespace cg = cooperative_groups;

namespace mh {

namespace {

constexpr int kResThreads = 1024;
constexpr int kResMaxBlocks = 256;
constexpr int kResCluster = 16;    // blocks of a cluster at most

struct ResArgs {
    const int64_t *slice_off;
    const int32_t *diag_slot;
    const int32_t *blk_slice;  // [n_blocks + 1] first slice of each block
    const int32_t *halo_off;   // [n_blocks + 1] first halo row of each block
    const int32_t *halo_row;   // halo rows of each block
    const uint16_t *idx;       // off-diagonal slots (slice by slice): index into own | halo entries
    InstCtl *ctl;
    double2 *part;             // [2][n_blocks][4] (sum, tag)
    unsigned long long *tag0;  // the launch's first tag; block 0 leaves the next launch's
    int32_t rows_cap;          // rows of the largest block (cluster)
    int32_t polls;             // of one value at most, before a block gives up
    int32_t *n_done;
    int32_t *err;
};

// (value, tag) in one single-copy atomic access (16 bytes for FP64, 8 for FP32): a tag that
// matches brings its value with it.  A buffer is overwritten whole at every second exchange, so
// the low 32 bits of the tag cannot meet an equal old one.
template <typename T> struct Tagged;
template <> struct Tagged<double> { using type = double2; };
template <> struct Tagged<float> { using type = float2; };

__device__ __forceinline__ void st_pair(float2 *p, float v, unsigned long long tag) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p),
                 "l"((unsigned long long)__float_as_uint(v) | tag << 32)
                 : "memory");
}
__device__ __forceinline__ float ld_pair(const float2 *p, unsigned long long want, bool &fresh) {
    unsigned long long u;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(u) : "l"(p) : "memory");
    fresh = (unsigned int)(u >> 32) == (unsigned int)want;
    return __uint_as_float((unsigned int)u);
}
__device__ __forceinline__ void st_pair(double2 *p, double v, unsigned long long tag) {
    asm volatile(
        "{\n\t.reg .b128 t;\n\t"
        "mov.b128 t, {%1, %2};\n\t"
        "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
        "l"(__double_as_longlong(v)), "l"(tag)
        : "memory");
}
__device__ __forceinline__ double ld_pair(const double2 *p, unsigned long long want, bool &fresh) {
    long long v;
    unsigned long long tag;
    asm volatile(
        "{\n\t.reg .b128 t;\n\t"
        "ld.relaxed.gpu.global.b128 t, [%2];\n\t"
        "mov.b128 {%0, %1}, t;\n\t}"
        : "=l"(v), "=l"(tag)
        : "l"(p)
        : "memory");
    fresh = tag == want;
    return __longlong_as_double(v);
}
// polls one value, at most `polls` times (late: it never came)
template <typename P, typename T>
__device__ __forceinline__ T await_pair(const P *p, T first, bool fresh, unsigned long long want, int polls, int &late) {
    for (int spin = 0; !fresh && !late && spin < polls; ++spin) first = ld_pair(p, want, fresh);
    late |= !fresh;
    return first;
}

// Sums four values over a warp; the sum of v[k] ends up in lanes 8k .. 8k + 7.
__device__ __forceinline__ double warp_sum4(const double (&v)[4], int lane) {
    const bool hi = lane & 16, up = lane & 8;
    const double a = (hi ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, hi ? v[0] : v[2], 16);
    const double b = (hi ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, hi ? v[1] : v[3], 16);
    double s = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// r - alpha q and the new direction, written with explicit fma: owner and halo copies must agree
// bit for bit
template <typename T> __device__ __forceinline__ void cg_step(T q, double alpha, double beta, T &r, T &p) {
    const double rr = fma(-alpha, (double)q, (double)r);
    p = (T)fma(beta, (double)p, rr);
    r = (T)rr;
}

// The run's scalars; only warp 0 works on them.  REG: rho, rr, tol2 and the counts in registers, which
// saves 0.15 us an iteration of loads in a serial chain, but costs every thread ten of the 64 that 1024
// threads have.  The chip-wide kernels spill there: 32 bytes (FP64) and 16 (FP32) with two rows a thread,
// 44 with three (FP64), 68 and 40 with four; those of three and four go without REG (n = 35 FP32: 8.0 us
// an iteration with it against 7.6).
struct RunState {
    double rho, rr, alpha, beta, tol2;
    int iter0, max_it, state;  // state 0: go on, 1: converged, 2: iteration cap, 3: breakdown, 4: not finite
};
template <bool REG> __device__ __forceinline__ void run_begin(RunState &st, const InstCtl *c) {
    if (!REG && threadIdx.x != 0) return;
    st.rho = c->rho;
    st.rr = c->rr;
    st.tol2 = c->tol2;
    st.iter0 = c->iter;
    st.max_it = c->max_it;
}
// What the sums of exchange x_no say: whether the run ended with the last update, else alpha and
// beta, which go to `out` in shared memory.  Called by warp 0 with the same sums in every lane.
template <bool REG>
__device__ __forceinline__ void run_step(RunState &st, RunState &out, double pq, double rq, double qq, double rr,
                                         unsigned int x_no) {
    double rho = st.rho, alpha = 0.0, beta = 0.0;
    int state = 0;
    if (x_no > 0) {
        rho = rr;
        if (!isfinite(rr)) state = 4;
        else if (rr <= st.tol2) state = 1;
        else if (st.iter0 + (int)x_no >= st.max_it) state = 2;
    }
    if (state == 0) {
        if (rho == 0.0) {
            state = 1;
        } else if (!(pq > 0.0) || !isfinite(pq)) {
            state = isfinite(pq) ? 3 : 4;
        } else {
            alpha = rho / pq;
            double rho_new = rho - 2.0 * alpha * rq + alpha * alpha * qq;
            if (rho_new < 0.0) rho_new = 0.0;
            beta = rho_new / rho;
        }
    }
    __syncwarp();
    const bool first = (threadIdx.x & 31) == 0;
    if (x_no > 0 && (REG || first)) st.rho = st.rr = rho;
    if (!first) return;
    out.alpha = alpha;
    out.beta = beta;
    out.state = state;
}
// thread 0 of block 0, behind its block's last barrier
__device__ __forceinline__ void run_end(const RunState &st, const RunState &out, InstCtl *c, int32_t *n_done,
                                        unsigned int x_no) {
    const int state = out.state;
    c->rho = st.rho;
    c->rr = st.rr;
    c->alpha = out.alpha;
    c->beta = out.beta;
    c->iter = st.iter0 + (int)x_no;
    c->status = state == 1 ? 0 : state == 2 ? 1 : state == 3 ? -8 : state ? -6 : 0;
    c->done = 1;
    atomicAdd(n_done, 1);
}

// The parts of a block's rows in shared memory.
template <typename T> struct ResRows {
    int s0, ns, nr, nh, n_off;
    int r0;
    T *sv, *sd, *sp, *hr;  // off-diagonal values; diagonal; p own | halo; r of the halo
    int32_t *hrow, *so;    // rows of the halo; first slot of each slice [ns + 1]
    uint16_t *si;          // column indices
};
template <typename T> __device__ __forceinline__ ResRows<T> res_rows(const ResArgs &a, unsigned char *sm) {
    ResRows<T> R;
    R.s0 = a.blk_slice[blockIdx.x];
    R.ns = a.blk_slice[blockIdx.x + 1] - R.s0;
    R.nh = a.halo_off[blockIdx.x + 1] - a.halo_off[blockIdx.x];
    R.nr = R.ns * kSliceRows;
    R.r0 = R.s0 * kSliceRows;
    R.n_off = (int)(a.slice_off[R.s0 + R.ns] - a.slice_off[R.s0]) - R.nr;
    R.sv = reinterpret_cast<T *>(sm);
    R.sd = R.sv + R.n_off;
    R.sp = R.sd + R.nr;
    R.hr = R.sp + R.nr + R.nh;
    R.hrow = reinterpret_cast<int32_t *>(R.hr + R.nh);
    R.so = R.hrow + R.nh;
    R.si = reinterpret_cast<uint16_t *>(R.so + R.ns + 1);
    return R;
}
// fills them (and x, r of the thread's rows) from global memory
template <typename T, int KR>
__device__ __forceinline__ void res_load(const ResArgs &a, const ResRows<T> &R, const T *__restrict__ val, const T *gx,
                                         const T *gr, const T *gp, T (&x)[KR], T (&r)[KR]) {
    const int lane = threadIdx.x & 31;
    const int64_t base = a.slice_off[R.s0];
    const int h0 = a.halo_off[blockIdx.x];
    for (int k = threadIdx.x; k <= R.ns; k += blockDim.x) R.so[k] = (int)(a.slice_off[R.s0 + k] - base) - kSliceRows * k;
    for (int k = threadIdx.x; k < R.n_off; k += blockDim.x) R.si[k] = a.idx[base - R.r0 + k];
    for (int k = threadIdx.x; k < R.nh; k += blockDim.x) {
        const int32_t row = a.halo_row[h0 + k];
        R.hrow[k] = row;
        R.hr[k] = gr[row];
        R.sp[R.nr + k] = gp[row];
    }
#pragma unroll
    for (int i = 0; i < KR; ++i) {
        const int lr = threadIdx.x + i * blockDim.x;
        x[i] = r[i] = (T)0;
        if (lr >= R.nr) continue;
        const int64_t row = R.r0 + lr, off = a.slice_off[R.s0 + (lr >> 5)];
        const int w = (int)((a.slice_off[R.s0 + (lr >> 5) + 1] - off) / kSliceRows);
        const int ds = a.diag_slot[row];
        int k = (int)(off - base) - kSliceRows * (lr >> 5) + lane;
        for (int j = 0; j < w; ++j) {
            const int64_t slot = off + (int64_t)j * kSliceRows + lane;
            const T v = val[slot];
            if (slot == ds) {
                R.sd[lr] = v;
            } else {
                R.sv[k] = v;
                k += kSliceRows;
            }
        }
        x[i] = gx[row];
        r[i] = gr[row];
        R.sp[lr] = gp[row];
    }
}
// (S^ p) of one of its rows
template <typename T> __device__ __forceinline__ double res_product(const ResRows<T> &R, int lr) {
    const int b = R.so[lr >> 5] + (threadIdx.x & 31), e = R.so[(lr >> 5) + 1];
    double y = (double)R.sd[lr] * (double)R.sp[lr];
#pragma unroll 6
    for (int k = b; k < e; k += kSliceRows) y = fma((double)R.sv[k], (double)R.sp[R.si[k]], y);
    return y;
}

// KR: rows per thread (x, r, q of the block's rows live in registers)
template <typename T, int KR>
__global__ void __launch_bounds__(kResThreads, 1)
    k_cg_resident(ResArgs a, const T *__restrict__ val, T *__restrict__ gx, T *__restrict__ gr, T *__restrict__ gp,
                  typename Tagged<T>::type *gq0, typename Tagged<T>::type *gq1) {
    InstCtl *c = a.ctl;
    if (c->done) return;  // the same value in every block: it is written after the last exchange
    extern __shared__ __align__(16) unsigned char rsm[];
    __shared__ double sh[32][4], gath[4][kResMaxBlocks];
    __shared__ RunState out;
    constexpr bool kReg = KR <= 2;
    RunState own;
    RunState &st = kReg ? own : out;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
    const int nb = (int)gridDim.x;
    const ResRows<T> R = res_rows<T>(a, rsm);
    const int nr = R.nr, nh = R.nh;
    const int r0 = R.r0;
    T *const sp = R.sp, *const hr = R.hr;
    const int32_t *const hrow = R.hrow;
    T x[KR], r[KR], q[KR];
    res_load<T, KR>(a, R, val, gx, gr, gp, x, r);
    run_begin<kReg>(st, c);
    if (threadIdx.x == 0) out.state = 0;
    double rr_part = 0.0;
    __syncthreads();
    const unsigned long long tag0 = *a.tag0;
    unsigned int x_no = 0;
    bool ok = true;
    for (;; ++x_no) {
        // A
        typename Tagged<T>::type *gq = (x_no & 1) ? gq1 : gq0;
        const unsigned long long tag = tag0 + x_no;
        double s[4] = {0.0, 0.0, 0.0, rr_part};
#pragma unroll
        for (int i = 0; i < KR; ++i) {
            const int lr = threadIdx.x + i * blockDim.x;
            if (lr >= nr) continue;
            const T pr = sp[lr];
            const double y = res_product(R, lr);
            q[i] = (T)y;
            st_pair(gq + (r0 + lr), q[i], tag);
            s[0] += (double)pr * y;
            s[1] += (double)r[i] * y;
            s[2] += y * y;
        }
        // X
        double w4 = warp_sum4(s, lane);
        if ((lane & 7) == 0) sh[warp][lane >> 3] = w4;
        __syncthreads();
        double2 *part = a.part + (x_no & 1) * 4 * (size_t)nb;
        if (warp == 0) {
            double t[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = lane < nw ? sh[lane][k] : 0.0;
            w4 = warp_sum4(t, lane);
            if ((lane & 7) == 0) st_pair(part + 4 * (size_t)blockIdx.x + (lane >> 3), w4, tag);
        }
        // the halo's q and the blocks' sums: the first loads of all are in flight together
        int late = 0;
        constexpr int kH = 3;
        T hq[kH];
        bool hf[kH];
#pragma unroll
        for (int i = 0; i < kH; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            hf[i] = true;
            hq[i] = k < nh ? ld_pair(gq + hrow[k], tag, hf[i]) : (T)0;
        }
        for (int k = threadIdx.x; k < 4 * nb; k += blockDim.x) {
            bool fresh;
            const double v = ld_pair(part + k, tag, fresh);
            gath[k & 3][k >> 2] = await_pair(part + k, v, fresh, tag, a.polls, late);
        }
#pragma unroll
        for (int i = 0; i < kH; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            if (k < nh) hq[i] = await_pair(gq + hrow[k], hq[i], hf[i], tag, a.polls, late);
        }
        ok = !__syncthreads_or(late);
        if (!ok) break;
        if (warp == 0) {
            double t[4] = {0.0, 0.0, 0.0, 0.0};
            for (int b = lane; b < nb; b += 32)
#pragma unroll
                for (int k = 0; k < 4; ++k) t[k] += gath[k][b];
            w4 = warp_sum4(t, lane);
            const double pq = __shfl_sync(0xffffffffu, w4, 0), rq = __shfl_sync(0xffffffffu, w4, 8),
                         qq = __shfl_sync(0xffffffffu, w4, 16), rr = __shfl_sync(0xffffffffu, w4, 24);
            run_step<kReg>(st, out, pq, rq, qq, rr, x_no);
        }
        __syncthreads();
        if (out.state) break;
        // B
        const double alpha = out.alpha, beta = out.beta;
#pragma unroll
        for (int i = 0; i < kH; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            if (k < nh) cg_step(hq[i], alpha, beta, hr[k], sp[nr + k]);
        }
        for (int k = threadIdx.x + kH * blockDim.x; k < nh; k += blockDim.x) {
            const T qh = await_pair(gq + hrow[k], (T)0, false, tag, a.polls, late);
            cg_step(qh, alpha, beta, hr[k], sp[nr + k]);
        }
        rr_part = 0.0;
#pragma unroll
        for (int i = 0; i < KR; ++i) {
            const int lr = threadIdx.x + i * blockDim.x;
            if (lr >= nr) continue;
            T ph = sp[lr];
            x[i] = (T)fma(alpha, (double)ph, (double)x[i]);
            cg_step(q[i], alpha, beta, r[i], ph);
            sp[lr] = ph;
            rr_part += (double)r[i] * (double)r[i];
        }
        ok = !__syncthreads_or(late);
        if (!ok) break;
    }
#pragma unroll
    for (int i = 0; i < KR; ++i) {
        const int lr = threadIdx.x + i * blockDim.x;
        if (lr >= nr) continue;
        gx[r0 + lr] = x[i];
        gr[r0 + lr] = r[i];
        gp[r0 + lr] = sp[lr];
    }
    if (threadIdx.x != 0) return;
    if (!ok) atomicExch(a.err, 1);
    if (blockIdx.x == 0) {
        *a.tag0 = tag0 + x_no + 2;
        run_end(st, out, c, a.n_done, x_no);
    }
}

// The same run by one thread-block cluster (kResCluster blocks at most), for the smallest systems:
// the exchange goes through distributed shared memory.  Every block writes its four sums into every
// block's mailbox and keeps its q in its own shared memory; after one cluster barrier the sums are
// there, and the halo's q is read from the owners.  Mailbox and q have two buffers, since a block can
// be one exchange ahead of another; the last barrier keeps every block until its q has been read.
// All blocks get the same sums, so they leave at the same exchange.
// What bounds it: the barrier and the chain of reductions around it; 16 SMs instead of up to 148
// also mean more rows on each.  Measured (B200, us an iteration, k_cg_resident -> this one): FP64,
// 1.1k edges 2.37 -> 1.74, 6.9k 2.83 -> 2.21, 13k 2.97 -> 2.70, 22k 2.79 -> 3.43; FP32 2.75 -> 2.42
// (3k), 3.31 -> 2.72 (6.9k), 3.41 -> 3.21 (13k), 3.36 -> 4.01 (22k).
template <typename T, int KR>
__global__ void __launch_bounds__(kResThreads, 1)
    k_cg_cluster(ResArgs a, const T *__restrict__ val, T *__restrict__ gx, T *__restrict__ gr, T *__restrict__ gp) {
    InstCtl *c = a.ctl;
    if (c->done) return;  // the same value in every block: it is written behind the last barrier
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) unsigned char rsm[];
    __shared__ double sh[32][4];
    __shared__ double2 mail[2][kResCluster][2];  // a block's four sums in two stores of 16 bytes
    __shared__ RunState out;
    constexpr bool kReg = KR <= 2;
    RunState own;
    RunState &st = kReg ? own : out;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
    const int nb = (int)gridDim.x;
    const int cap = a.rows_cap;  // q of a block: 2 x cap entries in front of its rows' parts, the same in every block
    T *sq = reinterpret_cast<T *>(rsm);
    const ResRows<T> R = res_rows<T>(a, rsm + 2 * (size_t)cap * sizeof(T));
    const int nr = R.nr, nh = R.nh;
    const int r0 = R.r0;
    T x[KR], r[KR], q[KR];
    res_load<T, KR>(a, R, val, gx, gr, gp, x, r);
    // the halo rows as (block, row of the block)
    for (int k = threadIdx.x; k < nh; k += blockDim.x) {
        const int sl = R.hrow[k] / kSliceRows;
        int b = 0;
        while (b + 1 < nb && a.blk_slice[b + 1] <= sl) ++b;
        R.hrow[k] = b << 16 | (R.hrow[k] - a.blk_slice[b] * kSliceRows);
    }
    run_begin<kReg>(st, c);
    if (threadIdx.x == 0) out.state = 0;
    double rr_part = 0.0;
    unsigned int x_no = 0;
    cl.sync();  // every block has started: its shared memory can be written
    for (;; ++x_no) {
        const int half = x_no & 1;
        double s[4] = {0.0, 0.0, 0.0, rr_part};
#pragma unroll
        for (int i = 0; i < KR; ++i) {
            const int lr = threadIdx.x + i * blockDim.x;
            if (lr >= nr) continue;
            const double pr = (double)R.sp[lr], y = res_product(R, lr);
            q[i] = (T)y;
            sq[half * cap + lr] = q[i];
            s[0] += pr * y;
            s[1] += (double)r[i] * y;
            s[2] += y * y;
        }
        double w4 = warp_sum4(s, lane);
        if ((lane & 7) == 0) sh[warp][lane >> 3] = w4;
        __syncthreads();
        if (warp == 0) {
            double t[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = lane < nw ? sh[lane][k] : 0.0;
            w4 = warp_sum4(t, lane);
#pragma unroll
            for (int k = 0; k < 4; ++k) t[k] = __shfl_sync(0xffffffffu, w4, 8 * k);
            if (lane < nb) {
                double2 *to = cl.map_shared_rank(&mail[half][blockIdx.x][0], lane);
                to[0] = make_double2(t[0], t[1]);
                to[1] = make_double2(t[2], t[3]);
            }
        }
        cl.sync();
        if (warp == 0) {
            const double2 none = make_double2(0.0, 0.0);
            const double2 m0 = lane < nb ? mail[half][lane][0] : none, m1 = lane < nb ? mail[half][lane][1] : none;
            const double t[4] = {m0.x, m0.y, m1.x, m1.y};
            w4 = warp_sum4(t, lane);
            const double pq = __shfl_sync(0xffffffffu, w4, 0), rq = __shfl_sync(0xffffffffu, w4, 8),
                         qq = __shfl_sync(0xffffffffu, w4, 16), rr = __shfl_sync(0xffffffffu, w4, 24);
            run_step<kReg>(st, out, pq, rq, qq, rr, x_no);
        }
        // the halo's q is on its way while warp 0 works out the scalars
        constexpr int kH = 2;
        T hq[kH];
#pragma unroll
        for (int i = 0; i < kH; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            hq[i] = (T)0;
            if (k < nh) hq[i] = cl.map_shared_rank(sq, R.hrow[k] >> 16)[half * cap + (R.hrow[k] & 0xffff)];
        }
        __syncthreads();
        if (out.state) break;
        const double alpha = out.alpha, beta = out.beta;
#pragma unroll
        for (int i = 0; i < kH; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            if (k < nh) cg_step(hq[i], alpha, beta, R.hr[k], R.sp[nr + k]);
        }
        for (int k = threadIdx.x + kH * blockDim.x; k < nh; k += blockDim.x)
            cg_step(cl.map_shared_rank(sq, R.hrow[k] >> 16)[half * cap + (R.hrow[k] & 0xffff)], alpha, beta, R.hr[k],
                    R.sp[nr + k]);
        rr_part = 0.0;
#pragma unroll
        for (int i = 0; i < KR; ++i) {
            const int lr = threadIdx.x + i * blockDim.x;
            if (lr >= nr) continue;
            T ph = R.sp[lr];
            x[i] = (T)fma(alpha, (double)ph, (double)x[i]);
            cg_step(q[i], alpha, beta, r[i], ph);
            R.sp[lr] = ph;
            rr_part += (double)r[i] * (double)r[i];
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < KR; ++i) {
        const int lr = threadIdx.x + i * blockDim.x;
        if (lr >= nr) continue;
        gx[r0 + lr] = x[i];
        gr[r0 + lr] = r[i];
        gp[r0 + lr] = R.sp[lr];
    }
    cl.sync();  // no block leaves while another may read its shared memory
    if (threadIdx.x == 0 && blockIdx.x == 0) run_end(st, out, c, a.n_done, x_no);
}

template <typename T> const void *cluster_kernel_of(int kr) {
    using K = void (*)(ResArgs, const T *, T *, T *, T *);
    const K k[4] = {k_cg_cluster<T, 1>, k_cg_cluster<T, 2>, k_cg_cluster<T, 3>, k_cg_cluster<T, 4>};
    return (const void *)k[kr - 1];
}
template <typename T> const void *kernel_of(int kr) {
    using Q = typename Tagged<T>::type;
    using K = void (*)(ResArgs, const T *, T *, T *, T *, Q *, Q *);
    const K k[4] = {k_cg_resident<T, 1>, k_cg_resident<T, 2>, k_cg_resident<T, 3>, k_cg_resident<T, 4>};
    return (const void *)k[kr - 1];
}
const void *kernel_of(const ResidentPlan &p) {
    if (p.cluster) return p.prec == 64 ? cluster_kernel_of<double>(p.kr) : cluster_kernel_of<float>(p.kr);
    return p.prec == 64 ? kernel_of<double>(p.kr) : kernel_of<float>(p.kr);
}

cudaLaunchConfig_t cluster_config(const ResidentPlan &plan, cudaLaunchAttribute *at, cudaStream_t s) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(plan.n_blocks);
    cfg.blockDim = dim3(plan.threads);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = plan.n_blocks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cfg;
}

// dynamic shared memory of a block with `slots` slots (diagonals included) in `ns` slices and nh
// halo rows
int64_t block_bytes(int64_t slots, int64_t ns, int64_t nh, int tsize) {
    const int64_t nr = ns * kSliceRows;
    return (slots - nr) * (tsize + 2) + nr * 2 * tsize + nh * (2 * tsize + 4) + (ns + 1) * 4 + 16;
}

}  // namespace

static bool plan_blocks(const std::vector<int64_t> &slice_off, const std::vector<int32_t> &col,
                        const std::vector<int32_t> &diag_slot, int prec, bool cluster, ResidentPlan &plan) {
    plan = ResidentPlan();
    plan.prec = prec;
    plan.cluster = cluster;
    const int64_t n_sl = (int64_t)slice_off.size() - 1;
    if (n_sl <= 0) return false;
    int dev = 0, sms = 0, optin = 0, coop = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop) {
        cudaGetLastError();
        return false;
    }
    const int tsize = prec == 64 ? 8 : 4;
    const int64_t limit = (int64_t)optin - 10240;  // the kernel's static shared memory: 9.3 KB
    if (block_bytes(slice_off[n_sl], n_sl, 0, tsize) > limit * sms) return false;
    int64_t nb = std::min<int64_t>(std::min(sms, kResMaxBlocks), (n_sl * kSliceRows + kResidentRows - 1) / kResidentRows);
    if (cluster) nb = kResCluster;
    nb = std::max<int64_t>(1, std::min(nb, n_sl));
    if (cluster)
        while (nb & (nb - 1)) nb &= nb - 1;  // powers of two
    // contiguous runs of slices, cut where the bytes before reach the block's share
    auto cost = [&](int64_t s) { return block_bytes(slice_off[s], s, 0, tsize); };
    const int64_t total = cost(n_sl);
    plan.blk_slice.assign(nb + 1, 0);
    int64_t s = 0, max_rows = 0;
    for (int64_t b = 0; b < nb; ++b) {
        plan.blk_slice[b] = (int32_t)s;
        const int64_t keep = nb - 1 - b;  // slices the later blocks need
        const int64_t upto = total * (b + 1) / nb;
        int64_t e = s + 1;
        while (e < n_sl - keep && cost(e) < upto) ++e;
        if (b == nb - 1) e = n_sl;
        max_rows = std::max(max_rows, (e - s) * kSliceRows);
        s = e;
    }
    plan.blk_slice[nb] = (int32_t)n_sl;
    if (max_rows > 4 * kResThreads) return false;
    plan.rows_cap = (int32_t)max_rows;
    // the halo of each block (its rows' columns in other blocks) and the 16-bit columns
    std::vector<std::vector<int32_t>> halo(nb);
    plan.idx.resize(slice_off[n_sl] - n_sl * kSliceRows);
    int fits = 1;
    int64_t smem = 0;
#pragma omp parallel for schedule(dynamic, 1) reduction(&& : fits) reduction(max : smem)
    for (int64_t b = 0; b < nb; ++b) {
        const int64_t f = plan.blk_slice[b], l = plan.blk_slice[b + 1], r0 = f * kSliceRows, r1 = l * kSliceRows;
        auto &h = halo[b];
        for (int64_t k = slice_off[f]; k < slice_off[l]; ++k)
            if (col[k] < r0 || col[k] >= r1) h.push_back(col[k]);
        std::sort(h.begin(), h.end());
        h.erase(std::unique(h.begin(), h.end()), h.end());
        const int64_t nr = r1 - r0, bytes = block_bytes(slice_off[l] - slice_off[f], l - f, (int64_t)h.size(), tsize) +
                                           (cluster ? 2 * max_rows * tsize : 0);
        smem = std::max(smem, bytes);
        fits = fits && bytes <= limit && nr + (int64_t)h.size() <= 65536;
        if (!fits) continue;
        for (int64_t sl = f; sl < l; ++sl) {
            const int64_t w = (slice_off[sl + 1] - slice_off[sl]) / kSliceRows;
            for (int64_t lane = 0; lane < kSliceRows; ++lane) {
                int64_t o = slice_off[sl] - sl * kSliceRows + lane;
                for (int64_t j = 0; j < w; ++j) {
                    const int64_t slot = slice_off[sl] + j * kSliceRows + lane;
                    if (slot == diag_slot[sl * kSliceRows + lane]) continue;
                    const int32_t cc = col[slot];
                    plan.idx[o] = (uint16_t)(cc >= r0 && cc < r1
                                                 ? cc - r0
                                                 : nr + (std::lower_bound(h.begin(), h.end(), cc) - h.begin()));
                    o += kSliceRows;
                }
            }
        }
    }
    if (!fits) return false;
    plan.halo_off.assign(nb + 1, 0);
    for (int64_t b = 0; b < nb; ++b) plan.halo_off[b + 1] = plan.halo_off[b] + (int32_t)halo[b].size();
    plan.halo_row.reserve(plan.halo_off[nb]);
    for (auto &h : halo) plan.halo_row.insert(plan.halo_row.end(), h.begin(), h.end());
    plan.smem = (size_t)smem;
    plan.n_blocks = (int)nb;
    plan.threads = (int)std::min<int64_t>(kResThreads, std::max<int64_t>(256, max_rows));
    plan.kr = (int)((max_rows + plan.threads - 1) / plan.threads);
    const void *k = kernel_of(plan);
    int fit = 0;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit);
    if (cluster) {
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = cluster_config(plan, at, nullptr);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&fit, k, &cfg);
    } else if (e == cudaSuccess) {
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&fit, k, plan.threads, plan.smem);
        fit = (int64_t)fit * sms >= nb;
    }
    if (e != cudaSuccess) cudaGetLastError();
    return e == cudaSuccess && fit > 0;
}

bool plan_resident(const std::vector<int64_t> &slice_off, const std::vector<int32_t> &col,
                   const std::vector<int32_t> &diag_slot, int prec, ResidentPlan &plan) {
    const int64_t rows = ((int64_t)slice_off.size() - 1) * kSliceRows;
    if (rows <= kClusterRows && plan_blocks(slice_off, col, diag_slot, prec, true, plan)) return true;
    return plan_blocks(slice_off, col, diag_slot, prec, false, plan);
}

cudaError_t launch_cg_resident(const DevSystem &sys, const ResidentPlan &plan, const ResidentDev &dev, int polls,
                               cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(dev.err, 0, sizeof(int32_t), s);
    if (e != cudaSuccess) return e;
    ResArgs a;
    a.slice_off = sys.slice_off;
    a.diag_slot = sys.diag_slot;
    a.blk_slice = dev.blk_slice;
    a.halo_off = dev.halo_off;
    a.halo_row = dev.halo_row;
    a.idx = dev.idx;
    a.ctl = sys.ctl;
    a.part = reinterpret_cast<double2 *>(dev.part);
    a.tag0 = dev.tag;
    a.n_done = sys.n_done;
    a.err = dev.err;
    const double *v64 = sys.val64;
    const float *v32 = sys.val32;
    double *x64 = sys.x, *r64 = sys.r, *p64 = sys.p;
    float *x32 = sys.x32, *r32 = sys.r32, *p32 = sys.p32;
    double2 *qd0 = reinterpret_cast<double2 *>(dev.q), *qd1 = qd0 + sys.n_rows;
    float2 *qf0 = reinterpret_cast<float2 *>(dev.q), *qf1 = qf0 + sys.n_rows;
    void *args64[] = {&a, &v64, &x64, &r64, &p64, &qd0, &qd1}, *args32[] = {&a, &v32, &x32, &r32, &p32, &qf0, &qf1};
    a.rows_cap = plan.rows_cap;
    a.polls = polls;
    if (plan.cluster) {
        cudaLaunchAttribute at[1];
        const cudaLaunchConfig_t cfg = cluster_config(plan, at, s);
        return cudaLaunchKernelExC(&cfg, kernel_of(plan), plan.prec == 64 ? args64 : args32);
    }
    return cudaLaunchCooperativeKernel(kernel_of(plan), dim3(plan.n_blocks), dim3(plan.threads),
                                       plan.prec == 64 ? args64 : args32, plan.smem, s);
}

}  // namespace mh
