// Flow post-processing on the device: the Darcy flux vector at every element centre from the
// side fluxes of the MH solution, DarcyFlowMHOutput::make_element_vector
// (src/flow/darcy_flow_mh_output.cc:301-323).  For each element E with sides s and side
// fluxes q_s, at the centre c (the mean of the nodes):
//     u_E = sum_s q_s RT0_s(c) / delta_E                          (delta_E: cross-section)
// with the lowest-order Raviart-Thomas basis of MHFEValues::RT0_value
// (src/flow/mh_fe_values.cc:76-118).  The reference evaluates the basis from its local-matrix
// parameters (line :150-152, triangle :193-211 with bas_func_0_triangle :293-301, tetrahedron
// :379-396); at the centre each of those equals
//     RT0_s(c) = (c - X_opp(s)) / (dim |E|)
// with X_opp(s) the node opposite side s (line: the other node; triangle: node (s+2) mod 3;
// tetrahedron: node s): |S_s| times the height of X_s over side s is dim |E|, the triangle
// formula is that vector written in the element's plane frame, and the line's is
// -(|v|/2) v / |v|^2 = (c - X_1) / |v| for side 0.  So
//     u_E = sum_s q_s (c - X_opp(s)) / (dim |E| delta_E),
// one division per element instead of the reference's per-side normals, square roots and
// divisions (which made the literal version FP64-divide bound: 172 us for 1.57M tetrahedra).
// The oracle (oracle/mh_oracle.c, orc_element_flux) keeps the reference's literal formulas,
// so the parity tests also check the identity.
// One thread per element, per-dimension element lists (no divergence between shapes); the
// output is [n_el][3], the three flux columns of the reference's raw output.
// Bytes per element: DIM+1 node indices and their coordinates (gathered, mostly from L2),
// DIM+1 side fluxes, the side offset, the cross-section and the list entry read, 24 written.
#include <cuda_runtime.h>

#include "device_system.hpp"
#include "mh_local.cuh"

namespace mh {
namespace {

template <int DIM>
__global__ void __launch_bounds__(128) k_element_flux(ElemData d, const int32_t *__restrict__ list, int64_t n,
                                                      const double *__restrict__ sol, double *__restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int e = list[t];
    constexpr int N = DIM + 1;
    V3 X[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int nd = d.el_nodes[4 * e + i];
        X[i] = {d.xyz[3 * nd], d.xyz[3 * nd + 1], d.xyz[3 * nd + 2]};
    }
    V3 c = {0.0, 0.0, 0.0};
#pragma unroll
    for (int i = 0; i < N; ++i) c = {c.x + X[i].x, c.y + X[i].y, c.z + X[i].z};
    c = v3scale(c, 1.0 / N);
    double dm;  // dim |E|
    if constexpr (DIM == 1) {
        dm = v3norm(v3sub(X[1], X[0]));
    } else if constexpr (DIM == 2) {
        dm = v3norm(v3cross(v3sub(X[1], X[0]), v3sub(X[2], X[0])));
    } else {
        dm = fabs(v3dot(v3cross(v3sub(X[1], X[0]), v3sub(X[2], X[0])), v3sub(X[3], X[0]))) / 2.0;
    }
    const double f = 1.0 / (dm * d.cross_section[e]);
    const int s0 = d.el_side_start[e];
    V3 u = {0.0, 0.0, 0.0};
#pragma unroll
    for (int s = 0; s < N; ++s) {
        const int opp = DIM == 1 ? 1 - s : DIM == 2 ? (s + 2) % 3 : s;
        const double q = sol[s0 + s];
        const V3 r = v3sub(c, X[opp]);
        u = {u.x + q * r.x, u.y + q * r.y, u.z + q * r.z};
    }
    out[3 * (int64_t)e] = u.x * f;
    out[3 * (int64_t)e + 1] = u.y * f;
    out[3 * (int64_t)e + 2] = u.z * f;
}

// ---- node pressures (make_node_scalar_param, darcy_flow_mh_output.cc:424-546) ---------------
// A node's pressure is the mean of the pressures of the elements and element sides that
// contain it, weighted by (1 - d / D) / (n - 1): d the distance from the node to that element's
// or side's centre, D the sum of those distances at the node, n their number.  The sums run over
// the node's elements (ascending, from a CSR incidence list built once per mesh): first every
// element centre, then every side of those elements that contains the node, the order in which
// the reference's two element loops reach the node.  No atomics: repeated calls give identical
// bits, and with the operation order of the reference (this file is compiled without FMA
// contraction) the result equals the FP64 restatement bit for bit.
//
// A thread per node is bound by the FP64 divisions and square roots of its 4 x 24 terms, twice over,
// in one chain.  A block takes 16 nodes instead: all its threads compute the distances (a thread
// per node and element: the centre and up to three sides) into shared memory, one lane per node adds
// them in order, all threads turn them into weighted pressures, one lane per node adds those in
// order.  Divisions by 3, by D and by n - 1 are products with the divisor's reciprocal and two
// corrections, which give the correctly rounded quotient (div_known).
// Measured (B200, 274,625 nodes of a cube with 1.57M tetrahedra): 848 -> 354 us, now bound by the instructions of
// the distances (about 300 a term) and the latency of their loads.
__device__ __forceinline__ double node_dist(V3 a, V3 b) {
    const V3 d = v3sub(a, b);
    return sqrt(d.x * d.x + d.y * d.y + d.z * d.z);
}

// a / b, correctly rounded, with y = 1 / b correctly rounded: two corrections of a y by fma.  The
// first leaves a quotient within one unit in the last place, the second rounds it correctly
// (P. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, IBM J.
// Res. Dev. 34, 1990, theorem 8).  Operands whose products could leave the normal range are divided.
__device__ __forceinline__ double div_known(double a, double b, double y) {
    const double m = fabs(a), n = fabs(b);
    if (!((m > 1e-140 && m < 1e140) && (n > 1e-140 && n < 1e140))) return a / b;
    double q = a * y;
    q = fma(fma(-b, q, a), y, q);
    return fma(fma(-b, q, a), y, q);
}

// the sum of N points divided by N
template <int N> __device__ __forceinline__ V3 mean_of(V3 c) {
    if (N == 3) {
        const double y = 1.0 / 3.0;
        return {div_known(c.x, 3.0, y), div_known(c.y, 3.0, y), div_known(c.z, 3.0, y)};
    }
    return v3scale(c, N == 4 ? 0.25 : N == 2 ? 0.5 : 1.0);  // exact
}

// whether side q of an element of dimension dim contains its node kv
__device__ __forceinline__ bool side_has(int dim, int q, int kv) {
    if (dim == 3) return q != kv;
    if (dim == 2) return dev_side_node(2, q, 0) == kv || dev_side_node(2, q, 1) == kv;
    return q == kv;
}

// one node and one of its elements: f(term, distance, index into sol) for the element's centre
// (term 0) and its sides that contain the node (terms 1, 2, ...); kv: the node's place in the element
template <int DIM, class F>
__device__ __forceinline__ void node_terms(const ElemData &d, int64_t v, int e, int s0, V3 Xv, int64_t n_sides,
                                           int64_t n_el, int &kv, F f) {
    constexpr int N = DIM + 1;
    const int4 nd4 = reinterpret_cast<const int4 *>(d.el_nodes)[e];
    const int nd[4] = {nd4.x, nd4.y, nd4.z, nd4.w};
    V3 X[N], c = {0.0, 0.0, 0.0};
    kv = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        if (nd[i] == v) kv = i;
        const double *x = d.xyz + 3 * (int64_t)nd[i];
        X[i] = {x[0], x[1], x[2]};
        c = {c.x + X[i].x, c.y + X[i].y, c.z + X[i].z};
    }
    f(0, node_dist(Xv, mean_of<N>(c)), n_sides + e);
    int t = 0;
#pragma unroll
    for (int q = 0; q < N; ++q) {
        bool has = false;
        V3 cs = {0.0, 0.0, 0.0};
#pragma unroll
        for (int k = 0; k < DIM; ++k) {
            const int m = dev_side_node(DIM, q, k);
            has |= m == kv;
            cs = {cs.x + X[m].x, cs.y + X[m].y, cs.z + X[m].z};
        }
        if (has) f(++t, node_dist(Xv, mean_of<DIM>(cs)), n_sides + n_el + d.side_edge[s0 + q]);
    }
}
// ... of any dimension; returns the element's dimension, which is also its number of such sides
template <class F>
__device__ __forceinline__ int node_terms_any(const ElemData &d, int64_t v, int e, V3 Xv, int64_t n_sides, int64_t n_el,
                                              int &kv, F f) {
    const int s0 = d.el_side_start[e], dim = d.el_side_start[e + 1] - s0 - 1;
    if (dim == 3) node_terms<3>(d, v, e, s0, Xv, n_sides, n_el, kv, f);
    else if (dim == 2) node_terms<2>(d, v, e, s0, Xv, n_sides, n_el, kv, f);
    else node_terms<1>(d, v, e, s0, Xv, n_sides, n_el, kv, f);
    return dim;
}

// the same by one thread (nodes of so many elements that a block's terms do not fit)
__device__ double node_pressure_serial(const ElemData &d, int64_t v, const int32_t *inc_el, int32_t p0, int32_t p1,
                                       const double *sol, int64_t n_sides, int64_t n_el) {
    const V3 Xv = {d.xyz[3 * v], d.xyz[3 * v + 1], d.xyz[3 * v + 2]};
    double D = 0.0, acc = 0.0;
    int cnt = 0, kv;
    for (int pass = 0; pass < 2; ++pass)
        for (int kind = 0; kind < 2; ++kind)
            for (int32_t q = p0; q < p1; ++q)
                node_terms_any(d, v, inc_el[q], Xv, n_sides, n_el, kv, [&](int t, double dist, int64_t at) {
                    if ((t > 0) != (kind > 0)) return;
                    if (pass == 0) {
                        D += dist;
                        ++cnt;
                    } else {
                        acc += sol[at] * (1.0 - dist / D) / (cnt - 1);
                    }
                });
    return acc;
}

// s plus the n side terms behind a pair's first, in order
__device__ __forceinline__ double add_sides(double s, const double *pair, int n) {
    const double a = pair[1], b = pair[2], c = pair[3];
    s += a;
    if (n > 1) s += b;
    if (n > 2) s += c;
    return s;
}

constexpr int kNpNodes = 16, kNpThreads = 128;
constexpr int kNpCap = 640;  // (node, element) pairs of a block: 16 nodes of 24 elements are 384
constexpr size_t kNpSmem = (4 * kNpCap + kNpNodes) * sizeof(double) + kNpCap;

__global__ void __launch_bounds__(kNpThreads, 8) k_node_pressure(ElemData d, const int32_t *__restrict__ inc_start,
                                                              const int32_t *__restrict__ inc_el, int64_t n_nodes,
                                                              const double *__restrict__ sol, int64_t n_sides,
                                                              int64_t n_el, double *__restrict__ out) {
    extern __shared__ double npm[];  // four terms per pair; one entry of padding per node (banks)
    unsigned char *terms = reinterpret_cast<unsigned char *>(npm + 4 * kNpCap + kNpNodes);
    __shared__ int32_t start[kNpNodes + 1];
    __shared__ double D[kNpNodes], yD[kNpNodes], n1[kNpNodes], yn1[kNpNodes];
    const int64_t v0 = (int64_t)blockIdx.x * kNpNodes;
    const int nn = (int)min((int64_t)kNpNodes, n_nodes - v0), t = threadIdx.x;
    if (t <= nn) start[t] = inc_start[v0 + t];
    __syncthreads();
    const int32_t first = start[0], pairs = start[nn] - first;
    if (pairs > kNpCap) {
        if (t < nn) out[v0 + t] = node_pressure_serial(d, v0 + t, inc_el, start[t], start[t + 1], sol, n_sides, n_el);
        return;
    }
    // eight threads to a node
    constexpr int kPer = kNpThreads / kNpNodes;
    const int k = t / kPer;
    const int64_t v = v0 + k;
    const int pa = k < nn ? start[k] - first + t % kPer : 0, pb = k < nn ? start[k + 1] - first : 0;
    for (int p = pa; p < pb; p += kPer) {
        const V3 Xv = {d.xyz[3 * v], d.xyz[3 * v + 1], d.xyz[3 * v + 2]};
        double *to = npm + 4 * p + k;
        int kv;
        const int dim = node_terms_any(d, v, inc_el[first + p], Xv, n_sides, n_el, kv,
                                       [&](int q, double dist, int64_t) { to[q] = dist; });
        terms[p] = (unsigned char)(dim | kv << 4);
    }
    __syncthreads();
    if (t < nn) {
        const int a = start[t] - first, b = start[t + 1] - first;
        double s = 0.0;
        int cnt = 0;
        for (int p = a; p < b; ++p) s += npm[4 * p + t];
        for (int p = a; p < b; ++p) {
            const int q = terms[p] & 15;
            cnt += 1 + q;
            s = add_sides(s, npm + 4 * p + t, q);
        }
        D[t] = s;
        yD[t] = 1.0 / s;
        n1[t] = (double)(cnt - 1);
        yn1[t] = 1.0 / n1[t];
    }
    __syncthreads();
    for (int p = pa; p < pb; p += kPer) {
        const int e = inc_el[first + p];
        const int dim = terms[p] & 15, kv = terms[p] >> 4, s0 = d.el_side_start[e];
        double *to = npm + 4 * p + k;
        auto weigh = [&](int q, int64_t at) {
            to[q] = div_known(sol[at] * (1.0 - div_known(to[q], D[k], yD[k])), n1[k], yn1[k]);
        };
        weigh(0, n_sides + e);
        for (int s = 0, q = 0; s <= dim; ++s)
            if (side_has(dim, s, kv)) weigh(++q, n_sides + n_el + d.side_edge[s0 + s]);
    }
    __syncthreads();
    if (t < nn) {
        const int a = start[t] - first, b = start[t + 1] - first;
        double s = 0.0;
        for (int p = a; p < b; ++p) s += npm[4 * p + t];
        for (int p = a; p < b; ++p) s = add_sides(s, npm + 4 * p + t, terms[p] & 15);
        out[v0 + t] = s;
    }
}

// ---- water balance (water_balance, darcy_flow_mh_output.cc:671-790) ----------------------------
// Per boundary region the sum of the outward side fluxes of its boundary objects, of the positive
// ones and of the negative ones; per bulk region the sum of |E| delta_E f_E.  The items (boundary
// sides, elements) come grouped by region in ascending order, cut into fixed chunks of at most
// kBalanceChunkItems items (host-built); one block per chunk sums it in a fixed order (strided
// per-thread sums, then a fixed tree), and one thread per region adds its chunks in order:
// deterministic, no atomics.

template <int NV> __device__ __forceinline__ void block_tree(double (&v)[NV], double (*sh)[NV]) {
    const int t = threadIdx.x;
#pragma unroll
    for (int k = 0; k < NV; ++k) sh[t][k] = v[k];
    __syncthreads();
    for (int w = blockDim.x / 2; w > 0; w >>= 1) {
        if (t < w)
#pragma unroll
            for (int k = 0; k < NV; ++k) sh[t][k] += sh[t + w][k];
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = sh[0][k];
}

// KIND 0: boundary sides (total, outflow, inflow); KIND 1: element sources
template <int KIND>
__global__ void __launch_bounds__(256) k_balance_chunks(ElemData d, const double *__restrict__ sol,
                                                        const int32_t *__restrict__ items,
                                                        const int64_t *__restrict__ chunk_begin,
                                                        double *__restrict__ partial) {
    constexpr int NV = KIND == 0 ? 3 : 1;
    __shared__ double sh[256][NV];
    const int64_t b0 = chunk_begin[blockIdx.x], b1 = chunk_begin[blockIdx.x + 1];
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = 0.0;
    for (int64_t t = b0 + threadIdx.x; t < b1; t += blockDim.x) {
        const int32_t it = items[t];
        if constexpr (KIND == 0) {
            const double q = sol[it];
            v[0] += q;
            if (q > 0.0) v[1] += q;
            else v[2] += q;
        } else {
            const int e = it;
            const double f = d.source[e];
            if (f == 0.0) continue;
            const int N = d.el_side_start[e + 1] - d.el_side_start[e];
            V3 X[4];
            for (int i = 0; i < N; ++i) {
                const int nd = d.el_nodes[4 * e + i];
                X[i] = {d.xyz[3 * nd], d.xyz[3 * nd + 1], d.xyz[3 * nd + 2]};
            }
            double meas;
            if (N == 2) {
                meas = v3norm(v3sub(X[1], X[0]));
            } else if (N == 3) {
                meas = v3norm(v3cross(v3sub(X[1], X[0]), v3sub(X[2], X[0]))) / 2.0;
            } else {
                meas = fabs(v3dot(v3cross(v3sub(X[1], X[0]), v3sub(X[2], X[0])), v3sub(X[3], X[0]))) / 6.0;
            }
            v[0] += meas * d.cross_section[e] * f;
        }
    }
    block_tree<NV>(v, sh);
    if (threadIdx.x == 0)
#pragma unroll
        for (int k = 0; k < NV; ++k) partial[(int64_t)blockIdx.x * NV + k] = v[k];
}

template <int NV>
__global__ void k_balance_regions(const int64_t *__restrict__ region_chunk, int32_t n_reg,
                                  const double *__restrict__ partial, double *__restrict__ out) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n_reg) return;
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = 0.0;
    for (int64_t c = region_chunk[r]; c < region_chunk[r + 1]; ++c)
#pragma unroll
        for (int k = 0; k < NV; ++k) v[k] += partial[c * NV + k];
#pragma unroll
    for (int k = 0; k < NV; ++k) out[(int64_t)r * NV + k] = v[k];
}

}  // namespace

cudaError_t launch_node_pressure(const ElemData &d, const int32_t *inc_start, const int32_t *inc_el, int64_t n_nodes,
                                 const double *sol, int64_t n_sides, int64_t n_el, double *out, cudaStream_t s) {
    if (n_nodes <= 0) return cudaSuccess;
    static_assert(kNpSmem <= 48 * 1024, "default limit of dynamic shared memory");
    k_node_pressure<<<(unsigned)((n_nodes + kNpNodes - 1) / kNpNodes), kNpThreads, kNpSmem, s>>>(
        d, inc_start, inc_el, n_nodes, sol, n_sides, n_el, out);
    return cudaGetLastError();
}

cudaError_t launch_water_balance(const ElemData &d, const double *sol, const BalanceLists &L, double *partial,
                                 double *bdr_out, double *src_out, cudaStream_t s) {
    if (L.n_bdr_chunks > 0)
        k_balance_chunks<0><<<(unsigned)L.n_bdr_chunks, 256, 0, s>>>(d, sol, L.bdr_items, L.bdr_chunk_begin, partial);
    k_balance_regions<3><<<(unsigned)((L.n_bdr_reg + 127) / 128), 128, 0, s>>>(L.bdr_region_chunk, L.n_bdr_reg, partial,
                                                                               bdr_out);
    double *sp = partial + 3 * L.n_bdr_chunks;
    if (L.n_src_chunks > 0)
        k_balance_chunks<1><<<(unsigned)L.n_src_chunks, 256, 0, s>>>(d, sol, L.src_items, L.src_chunk_begin, sp);
    k_balance_regions<1><<<(unsigned)((L.n_src_reg + 127) / 128), 128, 0, s>>>(L.src_region_chunk, L.n_src_reg, sp,
                                                                               src_out);
    return cudaGetLastError();
}

cudaError_t launch_element_flux(const ElemData &d, const DevAssembly &a, const double *sol, double *out,
                                cudaStream_t s) {
    auto blocks = [](int64_t n) { return (unsigned)((n + 127) / 128); };
    if (a.dim_count[1] > 0)
        k_element_flux<1><<<blocks(a.dim_count[1]), 128, 0, s>>>(d, a.dim_list[1], a.dim_count[1], sol, out);
    if (a.dim_count[2] > 0)
        k_element_flux<2><<<blocks(a.dim_count[2]), 128, 0, s>>>(d, a.dim_list[2], a.dim_count[2], sol, out);
    if (a.dim_count[3] > 0)
        k_element_flux<3><<<blocks(a.dim_count[3]), 128, 0, s>>>(d, a.dim_list[3], a.dim_count[3], sol, out);
    return cudaGetLastError();
}

}  // namespace mh
