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
// block that gives up sets *err and leaves.
// Measured (B200, us an iteration, two-kernel iteration -> this one): FP64, 6.9k edges 10.8 -> 2.8,
// 52k 11.7 -> 3.1, 175k 15.5 -> 4.6, 273k 17.7 -> 5.3; FP32, 52k 12.8 -> 3.5, 244k 17.1 -> 4.8,
// 528k 21.0 -> 7.5.  What is left is the exchange, about 2.2 us (two trips through L2, three block
// barriers), and from 200k edges on the FP64 arithmetic and conversions on the rows of one SM.
#include <algorithm>

#include <cuda_runtime.h>

#include "device_system.hpp"
#include "resident.hpp"

namespace mh {

namespace {

constexpr int kResThreads = 1024;
constexpr int kResMaxBlocks = 256;
constexpr int kResSpin = 1 << 21;  // polls of one value (about a second) before a block gives up

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
// polls one value, at most kResSpin times (late: it never came)
template <typename P, typename T>
__device__ __forceinline__ T await_pair(const P *p, T first, bool fresh, unsigned long long want, int &late) {
    for (int spin = 0; !fresh && !late && spin < kResSpin; ++spin) first = ld_pair(p, want, fresh);
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

// KR: rows per thread (x, r, q of the block's rows live in registers)
template <typename T, int KR>
__global__ void __launch_bounds__(kResThreads, 1)
    k_cg_resident(ResArgs a, const T *__restrict__ val, T *__restrict__ gx, T *__restrict__ gr, T *__restrict__ gp,
                  typename Tagged<T>::type *gq0, typename Tagged<T>::type *gq1) {
    InstCtl *c = a.ctl;
    if (c->done) return;  // the same value in every block: it is written after the last exchange
    extern __shared__ __align__(16) unsigned char rsm[];
    __shared__ double sh[32][4], gath[4][kResMaxBlocks], scal[2];
    __shared__ int s_state;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (int)(blockDim.x >> 5);
    const int nb = (int)gridDim.x;
    const int s0 = a.blk_slice[blockIdx.x], ns = a.blk_slice[blockIdx.x + 1] - s0;
    const int h0 = a.halo_off[blockIdx.x], nh = a.halo_off[blockIdx.x + 1] - h0;
    const int nr = ns * kSliceRows;
    const int64_t r0 = (int64_t)s0 * kSliceRows;
    const int64_t base = a.slice_off[s0];
    const int n_off = (int)(a.slice_off[s0 + ns] - base) - nr;  // off-diagonal slots
    T *sv = reinterpret_cast<T *>(rsm);                          // [n_off] values
    T *sd = sv + n_off, *sp = sd + nr, *hr = sp + nr + nh;       // diagonal; p own | halo; r of the halo
    int32_t *hrow = reinterpret_cast<int32_t *>(hr + nh);        // [nh] rows of the halo
    int32_t *so = hrow + nh;                                     // [ns + 1] first slot of each slice
    uint16_t *si = reinterpret_cast<uint16_t *>(so + ns + 1);    // [n_off] column indices
    for (int k = threadIdx.x; k <= ns; k += blockDim.x) so[k] = (int)(a.slice_off[s0 + k] - base) - kSliceRows * k;
    for (int k = threadIdx.x; k < n_off; k += blockDim.x) si[k] = a.idx[base - r0 + k];
    for (int k = threadIdx.x; k < nh; k += blockDim.x) {
        const int32_t row = a.halo_row[h0 + k];
        hrow[k] = row;
        hr[k] = gr[row];
        sp[nr + k] = gp[row];
    }
    T x[KR], r[KR], q[KR];
    double rr_part = 0.0;
#pragma unroll
    for (int i = 0; i < KR; ++i) {
        const int lr = threadIdx.x + i * blockDim.x;
        x[i] = r[i] = q[i] = (T)0;
        if (lr >= nr) continue;
        const int64_t row = r0 + lr, off = a.slice_off[s0 + (lr >> 5)];
        const int w = (int)((a.slice_off[s0 + (lr >> 5) + 1] - off) / kSliceRows);
        const int ds = a.diag_slot[row];
        int k = (int)(off - base) - kSliceRows * (lr >> 5) + lane;
        for (int j = 0; j < w; ++j) {
            const int64_t slot = off + (int64_t)j * kSliceRows + lane;
            const T v = val[slot];
            if (slot == ds) {
                sd[lr] = v;
            } else {
                sv[k] = v;
                k += kSliceRows;
            }
        }
        x[i] = gx[row];
        r[i] = gr[row];
        sp[lr] = gp[row];
    }
    __syncthreads();
    double rho = c->rho, rr_last = c->rr;
    const double tol2 = c->tol2;
    const int max_it = c->max_it;
    int iter = c->iter;
    const int iter0 = iter;
    const unsigned long long tag0 = *a.tag0;
    unsigned int x_no = 0;
    double alpha = 0.0, beta = 0.0;
    int status = 0;
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
            const int b = so[lr >> 5] + lane, e = so[(lr >> 5) + 1];
            const T pr = sp[lr];
            double y = (double)sd[lr] * (double)pr;
#pragma unroll 6
            for (int k = b; k < e; k += kSliceRows) y = fma((double)sv[k], (double)sp[si[k]], y);
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
            gath[k & 3][k >> 2] = await_pair(part + k, v, fresh, tag, late);
        }
#pragma unroll
        for (int i = 0; i < kH; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            if (k < nh) hq[i] = await_pair(gq + hrow[k], hq[i], hf[i], tag, late);
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
            int state = 0;  // 0: go on, 1: converged, 2: iteration cap, 3: breakdown, 4: not finite
            if (x_no > 0) {
                rho = rr_last = rr;
                if (!isfinite(rr)) state = 4;
                else if (rr <= tol2) state = 1;
                else if (iter0 + (int)x_no >= max_it) state = 2;
            }
            alpha = beta = 0.0;
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
            if (lane == 0) {
                scal[0] = alpha;
                scal[1] = beta;
                s_state = state;
            }
        }
        __syncthreads();
        iter = iter0 + (int)x_no;
        const int state = s_state;
        if (state) {
            status = state == 1 ? 0 : state == 2 ? 1 : state == 3 ? -8 : -6;
            break;
        }
        // B
        alpha = scal[0];
        beta = scal[1];
#pragma unroll
        for (int i = 0; i < kH; ++i) {
            const int k = threadIdx.x + i * blockDim.x;
            if (k < nh) cg_step(hq[i], alpha, beta, hr[k], sp[nr + k]);
        }
        for (int k = threadIdx.x + kH * blockDim.x; k < nh; k += blockDim.x) {
            const T qh = await_pair(gq + hrow[k], (T)0, false, tag, late);
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
        c->rho = rho;
        c->rr = rr_last;
        c->alpha = alpha;
        c->beta = beta;
        c->iter = iter;
        c->status = status;
        c->done = 1;
        atomicAdd(a.n_done, 1);
    }
}

template <typename T> const void *kernel_of(int kr) {
    using Q = typename Tagged<T>::type;
    using K = void (*)(ResArgs, const T *, T *, T *, T *, Q *, Q *);
    const K k[4] = {k_cg_resident<T, 1>, k_cg_resident<T, 2>, k_cg_resident<T, 3>, k_cg_resident<T, 4>};
    return (const void *)k[kr - 1];
}
const void *kernel_of(const ResidentPlan &p) { return p.prec == 64 ? kernel_of<double>(p.kr) : kernel_of<float>(p.kr); }

// dynamic shared memory of a block with `slots` slots (diagonals included) in `ns` slices and nh
// halo rows
int64_t block_bytes(int64_t slots, int64_t ns, int64_t nh, int tsize) {
    const int64_t nr = ns * kSliceRows;
    return (slots - nr) * (tsize + 2) + nr * 2 * tsize + nh * (2 * tsize + 4) + (ns + 1) * 4 + 16;
}

}  // namespace

bool plan_resident(const std::vector<int64_t> &slice_off, const std::vector<int32_t> &col,
                   const std::vector<int32_t> &diag_slot, int prec, ResidentPlan &plan) {
    plan = ResidentPlan();
    plan.prec = prec;
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
    nb = std::max<int64_t>(1, std::min(nb, n_sl));
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
        const int64_t nr = r1 - r0, bytes = block_bytes(slice_off[l] - slice_off[f], l - f, (int64_t)h.size(), tsize);
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
    int per_sm = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)limit) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, plan.threads, plan.smem) != cudaSuccess ||
        (int64_t)per_sm * sms < nb) {
        cudaGetLastError();
        return false;
    }
    return true;
}

cudaError_t launch_cg_resident(const DevSystem &sys, const ResidentPlan &plan, const ResidentDev &dev, cudaStream_t s) {
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
    return cudaLaunchCooperativeKernel(kernel_of(plan), dim3(plan.n_blocks), dim3(plan.threads),
                                       plan.prec == 64 ? args64 : args32, plan.smem, s);
}

}  // namespace mh
