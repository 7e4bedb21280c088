// Host runtime behind the C ABI of mh_darcy.h: owns the mesh topology, the device buffers,
// the CUDA stream and the captured Krylov graphs, and drives the kernels of assembly.cu and
// solver.cu.  It plays the role of DarcyFlowMH_Steady::update_solution with n_schurs = 2
// (src/flow/darcy_flow_mh.cc:375-433) and of make_schur0/1/2 + solve_system + resolve.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <functional>
#include <limits>
#include <memory>
#include <random>
#include <new>
#include <string>
#include <vector>

#include "device_system.hpp"
#include "amg.hpp"
#include "learned.hpp"
#include "smoother_nn.hpp"
#include "mesh_store.hpp"
#include "resident.hpp"
#include "mh_darcy.h"
#include "system_build.hpp"
#include "topology.hpp"


enum class Pc { Nn, Cheb, Amg };  // preconditioners of the flexible-CG solve

struct FcgKey {  // what a captured flexible-CG graph depends on
    int kind = -1, ipg = 0, degree = 0;
    double lo = 0.0, hi = 0.0;
    int64_t amg_epoch = -1;
    bool prof = false;
    bool loop = false;  // the iterations sit in a device-side WHILE loop
    bool operator==(const FcgKey &o) const {
        return kind == o.kind && ipg == o.ipg && degree == o.degree && lo == o.lo && hi == o.hi &&
               amg_epoch == o.amg_epoch && prof == o.prof && loop == o.loop;
    }
};

struct mh_handle {
    mh::MeshData mesh;
    mh::Topology topo;
    mh::HostSystem hs;
    std::vector<int32_t> ngh_hi_el;
    std::vector<double> ngh_meas;
    bool device = false;
    int device_id = -1;
    cudaStream_t stream = nullptr;      // stream all work is issued on (own or caller's)
    cudaStream_t own_stream = nullptr;  // the handle's stream; CUDA graphs are captured on it
    std::vector<void *> allocs;
    mh::ElemData ed{};
    mh::DevSystem sys{};
    mh::DevAssembly as{};
    double *sol = nullptr, *sol_prev = nullptr;
    double *d_elflux = nullptr;         // element flux vectors for mh_get_element_flux (3 n_el)
    double *d_node_p = nullptr;                                // node pressures
    int32_t *d_node_inc_start = nullptr, *d_node_inc = nullptr;  // node -> elements (ascending)
    // water balance: items grouped by region and their chunks (built per call, capacities kept)
    int32_t *d_bal_items = nullptr;
    int64_t *d_bal_index = nullptr;     // chunk begins and region-chunk offsets of both kinds
    double *d_balance = nullptr;        // chunk partials, then the per-region sums
    int64_t bal_items_cap = 0, bal_index_cap = 0, balance_cap = 0;
    // convection matrix of the transport: pattern (built once), host copies of its CSR
    // structure, device values and porosity
    bool tr_built = false;
    mh::TransportPattern conv{};
    std::vector<int32_t> tr_row_ptr, tr_col;
    double *d_tr_val = nullptr, *d_tr_por = nullptr;
    double *d_aniso = nullptr;
    bool coeffs_set = false, bc_set = false, assembled = false, solved = false;
    bool general = false;               // a general SPD system given in CSR form (no mesh)
    double *d_csr_val = nullptr;        // its values in the caller's order, and their SELL slots
    int32_t *d_csr_slot = nullptr;
    bool rhs_stale = false;             // boundary values changed since the last assembly
    int time_mode = 0;
    double dt = 0.0;
    // captured Krylov iterations: [precision 64/32][plain / with per-kernel timing events]
    cudaGraphExec_t graph[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
    int graph_iters[2][2] = {{0, 0}, {0, 0}};
    // the same iterations in a conditional WHILE loop (one launch per Krylov run; per precision)
    cudaGraphExec_t loop_graph[2] = {nullptr, nullptr};
    int loop_iters[2] = {0, 0};
    int32_t *d_loop = nullptr;  // {bodies run, body cap} of the device-side loop
    // Krylov runs in shared memory (resident.cu), per precision 64/32: planned at the first run
    // (0: not yet, 1: usable, -1: the system does not fit)
    mh::ResidentPlan res_plan[2];
    int res_state[2] = {0, 0};
    mh::ResidentDev res_dev[2];
    int k1_group = 128;         // elements per K1 block (mh_autotune_ex)
    int amg_fine_passes = 0;    // pairing passes from the fine level chosen by mh_autotune_ex (0: default)
    bool host_loop = false;     // the current solve polls from the host instead (mh_solve_opts)
    bool loop_unavailable = false;  // the device-side loop could not be built: poll from the host
    std::vector<cudaEvent_t> prof_ev[2];
    int32_t *h_done = nullptr;
    void *h_small = nullptr;            // pinned staging of small read-backs (read_back)
    cudaEvent_t ev[8] = {};
    float ms_assembly = 0.f;
    int64_t n_launch = 0;               // kernels launched so far
    double kernel_ms[MH_KERNEL_CLASSES] = {};
    int32_t kernel_count[MH_KERNEL_CLASSES] = {};
    std::vector<int32_t> inst_iters, inst_status;  // per instance, last solve
    std::vector<double> inst_rel;
    // learned preconditioner: fp32 master weights, bf16 fragments, Adam state, work buffers
    // learned smoother network: parameters, Adam state, gradient; row features of the current
    // matrix and the activations of an inference pass; the weights it gives
    float *nn_w = nullptr, *nn_m = nullptr, *nn_v = nullptr, *nn_grad = nullptr;
    int nn_step = 0;
    float *sn_x = nullptr, *sn_w = nullptr;
    mh::SnActs sn_inf{};
    int64_t sn_x_epoch = -1;            // matrix epoch the features were computed from
    int64_t sn_key_epoch = -1;          // matrix epoch and training step of the weights in sn_w
    int sn_key_step = -1;
    bool user_fine_w = false;           // mh_smoother_weights_set holds weights in d_fine_w
    float *cheb_z0 = nullptr, *cheb_z1 = nullptr, *cheb_d = nullptr;
    unsigned int *spec_bound = nullptr;
    double *d_loss = nullptr;
    mh::Amg amg;                        // aggregation multigrid (MH_SOLVER_AMG)
    float *d_fine_w = nullptr;          // fine-level smoother weights per solver row (or unused)
    int64_t amg_epoch = 0;              // setups so far (captured graphs refer to one)
    int64_t matrix_epoch = 0;           // matrix assemblies so far
    int64_t amg_matrix_epoch = -1;      // the assembly the current hierarchy was built from
    std::vector<int32_t> bc_type_host;  // boundary data that enters the matrix, as last set
    std::vector<double> bc_sigma_host;
    cudaGraphExec_t fcg_graph = nullptr;
    FcgKey fcg_key{};
    std::vector<mh::AmgProf> amg_prof;  // timing events of the V-cycles of one FCG graph
    mh::SnActs sn_tr{};                 // activations of a training pass
    mh::SnScratch sn_sc{};
    float *tv[16] = {};                 // vectors of the smoother gradient
    double *tdot = nullptr;             // dot-product partials and results
    bool tr_ready = false;
    bool amg_training = false;          // the hierarchy is the training one ...
    int64_t tr_hier_epoch = -1;         // ... of this matrix epoch
    float *pair_r = nullptr, *pair_e = nullptr;  // training pairs, [cap][n_rows] each
    int pair_cap = 0;
    double *x_star = nullptr, *pair_acc = nullptr;
    double *x_keep = nullptr;  // the solution before a segment that may be undone (polish)
    std::string err;
};

namespace {

using mh::HostSystem;

#define CK(call)                                                                        \
    do {                                                                                \
        cudaError_t e_ = (call);                                                        \
        if (e_ != cudaSuccess) {                                                        \
            h->err = std::string(#call) + ": " + cudaGetErrorString(e_);                \
            cudaGetLastError(); /* clear a non-sticky error so later checks see fresh state */ \
            return MH_ERR_CUDA;                                                         \
        }                                                                               \
    } while (0)

// A read-back that the caller waits for.  Small ones go through pinned memory: a copy into
// pageable memory is staged by the driver and holds the caller several microseconds longer.
constexpr size_t kSmallBytes = 64 * 1024;
int read_back(mh_handle *h, void *dst, const void *src, size_t bytes) {
    const bool small = bytes <= kSmallBytes && h->h_small;
    CK(cudaMemcpyAsync(small ? h->h_small : dst, src, bytes, cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    if (small) std::memcpy(dst, h->h_small, bytes);
    return MH_OK;
}

template <class T> T *dalloc(mh_handle *h, size_t n) {
    void *p = nullptr;
    if (n == 0) n = 1;
    if (cudaMalloc(&p, n * sizeof(T)) != cudaSuccess) return nullptr;
    h->allocs.push_back(p);
    return (T *)p;
}

// On the handle's stream, which the legacy stream of the plain calls does not order (own_stream does
// not wait for it): what the handle launches next finds the data there.
template <class T> int upload(mh_handle *h, T *&dst, const std::vector<T> &src) {
    dst = dalloc<T>(h, src.size());
    if (!dst) {
        h->err = "cudaMalloc failed";
        return MH_ERR_NOMEM;
    }
    if (!src.empty())
        CK(cudaMemcpyAsync(dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice, h->stream));
    return MH_OK;
}

double side_measure_host(const mh::MeshData &m, int64_t e, int s) {
    int d = m.dim[e];
    if (d == 1) return 1.0;
    const double *X[3];
    for (int k = 0; k < d; ++k) X[k] = &m.xyz[3 * m.nodes[4 * e + mh::side_node(d, s, k)]];
    if (d == 2) {
        double dx = X[1][0] - X[0][0], dy = X[1][1] - X[0][1], dz = X[1][2] - X[0][2];
        return std::sqrt(dx * dx + dy * dy + dz * dz);
    }
    double u[3] = {X[1][0] - X[0][0], X[1][1] - X[0][1], X[1][2] - X[0][2]};
    double v[3] = {X[2][0] - X[0][0], X[2][1] - X[0][1], X[2][2] - X[0][2]};
    double c[3] = {u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]};
    return 0.5 * std::sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
}

__global__ void k_fill(double *dst, int64_t n, double v) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = v;
}

__global__ void k_scatter(int64_t n, const int32_t *__restrict__ to, const double *__restrict__ v,
                          double *__restrict__ dst) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[to[i]] = v[i];
}

int device_setup(mh_handle *h) {
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || n_dev == 0) {
        cudaGetLastError();
        h->device = false;
        return MH_OK;
    }
    CK(cudaGetDevice(&h->device_id));
    CK(cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking));
    h->stream = h->own_stream;
    for (auto &e : h->ev) CK(cudaEventCreate(&e));
    CK(cudaHostAlloc((void **)&h->h_done, sizeof(int32_t) * 4, cudaHostAllocDefault));
    CK(cudaHostAlloc(&h->h_small, kSmallBytes, cudaHostAllocDefault));
    const mh::MeshData &m = h->mesh;
    const mh::Topology &t = h->topo;
    const HostSystem &hs = h->hs;
    int rc;
    double *xyz;
    int32_t *el_nodes, *el_side_start, *side_edge, *side_bdr, *el_ngh_start, *el_ngh, *ngh_edge, *ngh_hi;
    double *ngh_meas;
    if ((rc = upload(h, xyz, m.xyz)) || (rc = upload(h, el_nodes, m.nodes)) ||
        (rc = upload(h, el_side_start, t.el_side_start)) || (rc = upload(h, side_edge, t.side_edge)) ||
        (rc = upload(h, side_bdr, t.side_bdr)) || (rc = upload(h, el_ngh_start, t.el_ngh_start)) ||
        (rc = upload(h, el_ngh, t.el_ngh)) || (rc = upload(h, ngh_edge, t.ngh_edge)) ||
        (rc = upload(h, ngh_hi, h->ngh_hi_el)) || (rc = upload(h, ngh_meas, h->ngh_meas)))
        return rc;
    mh::ElemData &d = h->ed;
    d.xyz = xyz;
    d.el_nodes = el_nodes;
    d.el_side_start = el_side_start;
    d.side_edge = side_edge;
    d.side_bdr = side_bdr;
    d.el_ngh_start = el_ngh_start;
    d.el_ngh = el_ngh;
    d.ngh_edge = ngh_edge;
    d.ngh_hi_el = ngh_hi;
    d.ngh_side_measure = ngh_meas;
    const int64_t n_el = m.n_el, n_bdr = t.n_bdr();
    double *cond = dalloc<double>(h, n_el), *cs = dalloc<double>(h, n_el), *sg = dalloc<double>(h, n_el);
    double *src = dalloc<double>(h, n_el), *sto = dalloc<double>(h, n_el);
    int32_t *bct = dalloc<int32_t>(h, n_bdr);
    double *bcp = dalloc<double>(h, n_bdr), *bcf = dalloc<double>(h, n_bdr), *bcs = dalloc<double>(h, n_bdr);
    if (!cond || !cs || !sg || !src || !sto || !bct || !bcp || !bcf || !bcs) return MH_ERR_NOMEM;
    d.conductivity = cond;
    d.cross_section = cs;
    d.sigma = sg;
    d.source = src;
    d.storativity = sto;
    d.anisotropy = nullptr;
    d.bc_type = bct;
    d.bc_pressure = bcp;
    d.bc_flux = bcf;
    d.bc_sigma = bcs;
    d.time_mode = 0;
    d.dt = 1.0;

    mh::DevAssembly &a = h->as;
    a.n_blk = hs.n_blk;
    a.n_rhs_loc = hs.n_rhs_loc;
    if ((rc = upload(h, a.blk_off, hs.blk_off)) || (rc = upload(h, a.rhs_off, hs.rhs_off)) ||
        (rc = upload(h, a.slot_cstart, hs.slot_cstart)) || (rc = upload(h, a.slot_cidx, hs.slot_cidx)) ||
        (rc = upload(h, a.row_cstart, hs.row_cstart)) || (rc = upload(h, a.row_cidx, hs.row_cidx)))
        return rc;
    for (int dd = 1; dd <= 3; ++dd) {
        a.dim_count[dd] = (int64_t)hs.dim_list[dd].size();
        if ((rc = upload(h, a.dim_list[dd], hs.dim_list[dd]))) return rc;
    }
    a.n_add = (int64_t)hs.add_slot.size();
    if (a.n_add > 0 && ((rc = upload(h, a.add_slot, hs.add_slot)) || (rc = upload(h, a.add_val, hs.add_val)))) return rc;
    a.blk = dalloc<double>(h, hs.n_blk);
    a.rhs_loc = dalloc<double>(h, hs.n_rhs_loc);
    a.status = dalloc<int32_t>(h, 1);
    if (!a.blk || !a.rhs_loc || !a.status) return MH_ERR_NOMEM;

    mh::DevSystem &s = h->sys;
    s.n_rows = hs.n_rows;
    s.n_slices = hs.n_slices;
    s.n_tiles = hs.n_tiles;
    s.n_slots = hs.n_slots;
    s.rows_per_thread = hs.rows_per_thread;
    s.n_inst = (int32_t)hs.inst_el.size() - 1;
    if ((rc = upload(h, s.slice_off, hs.slice_off)) || (rc = upload(h, s.col, hs.sell_col)) ||
        (rc = upload(h, s.diag_slot, hs.diag_slot)) || (rc = upload(h, s.row_edge, hs.row_edge)) ||
        (rc = upload(h, s.edge_row, hs.edge_row)) || (rc = upload(h, s.tile_inst, hs.tile_inst)))
        return rc;
    int32_t max_blocks = 1;
    for (int k = 0; k < 2; ++k) {
        mh::DevPlan &dp = s.plan[k];
        const auto &hp = hs.plan[k];
        dp.n_blocks = (int32_t)hp.blk_inst.size();
        max_blocks = std::max(max_blocks, dp.n_blocks);
        if ((rc = upload(h, dp.blk_inst, hp.blk_inst)) || (rc = upload(h, dp.tile_begin, hp.blk_tile_begin)) ||
            (rc = upload(h, dp.tile_end, hp.blk_tile_end)) || (rc = upload(h, dp.inst_blk, hp.inst_blk)))
            return rc;
    }
    const int64_t nr = hs.n_rows;
    s.val_raw = dalloc<double>(h, hs.n_slots);
    s.val64 = dalloc<double>(h, hs.n_slots);
    s.val32 = dalloc<float>(h, hs.n_slots);
    s.dsq = dalloc<double>(h, nr);
    s.b = dalloc<double>(h, nr);
    s.bh = dalloc<double>(h, nr);
    s.x = dalloc<double>(h, nr);
    s.r = dalloc<double>(h, nr);
    s.p = dalloc<double>(h, nr);
    s.q = dalloc<double>(h, nr);
    s.s = dalloc<double>(h, nr);
    s.x32 = dalloc<float>(h, nr);
    s.r32 = dalloc<float>(h, nr);
    s.p32 = dalloc<float>(h, nr);
    s.q32 = dalloc<float>(h, nr);
    s.z32 = dalloc<float>(h, nr);
    s.partial = dalloc<double>(h, (size_t)max_blocks * 4);
    s.ctl = dalloc<mh::InstCtl>(h, s.n_inst);
    s.n_done = dalloc<int32_t>(h, 1);
    s.inst_sums = dalloc<double>(h, mh::kSumStride * (size_t)s.n_inst);
    s.sum_ticket = dalloc<uint32_t>(h, s.n_inst);
    if (!s.val_raw || !s.val64 || !s.val32 || !s.dsq || !s.b || !s.bh || !s.x || !s.r || !s.p || !s.q || !s.s ||
        !s.x32 || !s.r32 || !s.p32 || !s.q32 || !s.z32 || !s.partial || !s.ctl || !s.n_done || !s.inst_sums ||
        !s.sum_ticket)
        return MH_ERR_NOMEM;
    std::vector<mh::InstCtl> ctl(s.n_inst);
    for (int i = 0; i < s.n_inst; ++i) {
        std::memset(&ctl[i], 0, sizeof(mh::InstCtl));
        ctl[i].done = 1;
    }
    CK(cudaMemcpyAsync(s.ctl, ctl.data(), sizeof(mh::InstCtl) * ctl.size(), cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemsetAsync(s.x, 0, nr * sizeof(double), h->stream));
    CK(cudaMemsetAsync(s.x32, 0, nr * sizeof(float), h->stream));
    CK(cudaMemsetAsync(s.sum_ticket, 0, s.n_inst * sizeof(uint32_t), h->stream));
    CK(cudaMemsetAsync(s.inst_sums, 0, mh::kSumStride * s.n_inst * sizeof(double), h->stream));
    if (h->general) {
        // the slots outside the caller's pattern hold a unit diagonal (padding rows) or 0 for good
        if ((rc = upload(h, h->d_csr_slot, hs.csr_slot))) return rc;
        h->d_csr_val = dalloc<double>(h, hs.nnz);
        if (!h->d_csr_val) return MH_ERR_NOMEM;
        CK(cudaMemsetAsync(s.val_raw, 0, hs.n_slots * sizeof(double), h->stream));
        CK(cudaMemsetAsync(s.b, 0, nr * sizeof(double), h->stream));
        const int64_t n_pad = nr - t.n_edges();
        if (n_pad > 0) {
            // s.p is the staging: nothing has been solved yet
            k_fill<<<(unsigned)((n_pad + 255) / 256), 256, 0, h->stream>>>(s.p, n_pad, 1.0);
            k_scatter<<<(unsigned)((n_pad + 255) / 256), 256, 0, h->stream>>>(n_pad, s.diag_slot + t.n_edges(), s.p,
                                                                              s.val_raw);
            CK(cudaGetLastError());
        }
    }
    const int64_t msize = t.n_sides() + m.n_el + t.n_edges();
    h->sol = dalloc<double>(h, msize);
    h->sol_prev = dalloc<double>(h, msize);
    h->d_loop = dalloc<int32_t>(h, 2);
    if (!h->sol || !h->sol_prev || !h->d_loop) return MH_ERR_NOMEM;
    CK(cudaMemsetAsync(h->sol, 0, msize * sizeof(double), h->stream));
    CK(cudaMemsetAsync(h->sol_prev, 0, msize * sizeof(double), h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->device = true;
    return MH_OK;
}

// Switches rows per thread and the block plans (matrix layout unchanged) and drops the
// captured graphs, which hold the old launch shape.
int apply_launch_shape(mh_handle *h, int R, const int targets[2]) {
    CK(cudaStreamSynchronize(h->stream));
    mh::set_launch_shape(h->hs, R, targets);
    const HostSystem &hs = h->hs;
    mh::DevSystem &s = h->sys;
    int rc;
    s.rows_per_thread = R;
    s.n_tiles = hs.n_tiles;
    if ((rc = upload(h, s.tile_inst, hs.tile_inst))) return rc;
    int32_t max_blocks = 1;
    for (int k = 0; k < 2; ++k) {
        mh::DevPlan &dp = s.plan[k];
        const auto &hp = hs.plan[k];
        dp.n_blocks = (int32_t)hp.blk_inst.size();
        max_blocks = std::max(max_blocks, dp.n_blocks);
        if ((rc = upload(h, dp.blk_inst, hp.blk_inst)) || (rc = upload(h, dp.tile_begin, hp.blk_tile_begin)) ||
            (rc = upload(h, dp.tile_end, hp.blk_tile_end)) || (rc = upload(h, dp.inst_blk, hp.inst_blk)))
            return rc;
    }
    s.partial = dalloc<double>(h, (size_t)max_blocks * 4);
    if (!s.partial) return MH_ERR_NOMEM;
    for (auto &gp : h->graph)
        for (auto &g : gp)
            if (g) {
                cudaGraphExecDestroy(g);
                g = nullptr;
            }
    for (auto &gi : h->graph_iters) gi[0] = gi[1] = 0;
    for (auto &g : h->loop_graph)
        if (g) {
            cudaGraphExecDestroy(g);
            g = nullptr;
        }
    h->loop_iters[0] = h->loop_iters[1] = 0;
    if (h->fcg_graph) cudaGraphExecDestroy(h->fcg_graph);
    h->fcg_graph = nullptr;
    return MH_OK;
}

int need_device(mh_handle *h) {
    if (!h) return MH_ERR_INVALID;
    if (!h->device) {
        h->err = "no CUDA device";
        return MH_ERR_CUDA;
    }
    return MH_OK;
}

// input checks on the host threads (element fields of millions of entries are checked on
// every unsteady step)
int check_finite(const double *a, int64_t n) {
    if (!a) return 1;
    int ok = 1;
#pragma omp parallel for reduction(&& : ok) schedule(static) if (n > (1 << 16))
    for (int64_t i = 0; i < n; ++i) ok = ok && std::isfinite(a[i]);
    return ok;
}

int check_positive(const double *a, int64_t n) {
    if (!a) return 1;
    int ok = 1;
#pragma omp parallel for reduction(&& : ok) schedule(static) if (n > (1 << 16))
    for (int64_t i = 0; i < n; ++i) ok = ok && a[i] > 0.0;
    return ok;
}

// a field from the caller's host array, or its default value filled on the device
int fill_or_default(mh_handle *h, double *dst, const double *src, int64_t n, double dflt) {
    if (n <= 0) return MH_OK;
    if (src) {
        CK(cudaMemcpyAsync(dst, src, n * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    } else {
        k_fill<<<(unsigned)((n + 255) / 256), 256, 0, h->stream>>>(dst, n, dflt);
        CK(cudaGetLastError());
    }
    return MH_OK;
}

// Assembly on the device: K1 local blocks -> gather -> scaling.  mode 3 = matrix + rhs, 2 = rhs.
int assemble_impl(mh_handle *h, int mode) {
    h->ed.prev_pressure = h->sol_prev + h->topo.n_sides();
    h->ed.prev_edge = h->sol_prev + h->topo.n_sides() + h->mesh.n_el;
    CK(cudaMemsetAsync(h->as.status, 0, sizeof(int32_t), h->stream));
    CK(cudaEventRecord(h->ev[0], h->stream));
    CK(mh::launch_local_blocks(h->ed, h->as, mode, h->k1_group, h->stream));
    CK(mh::launch_gather(h->as, h->sys, mode, h->stream));
    CK(mh::launch_scale(h->sys, (mode & 1) ? 1 : 0, h->stream));
    CK(cudaEventRecord(h->ev[1], h->stream));
    for (int d = 1; d <= 3; ++d) h->n_launch += h->as.dim_count[d] > 0;
    h->n_launch += 1 + ((mode & 1) ? 3 : 1);
    int32_t st = 0;
    if (int rc = read_back(h, &st, h->as.status, sizeof(st))) return rc;
    CK(cudaEventElapsedTime(&h->ms_assembly, h->ev[0], h->ev[1]));
    if (st & 1) {
        h->err = "singular local MH matrix (|det| < DBL_MIN/DBL_EPSILON)";
        return MH_ERR_SINGULAR;
    }
    if (st & 2) {
        h->err = "non-finite value in the assembled system";
        return MH_ERR_NONFINITE;
    }
    if (mode & 2) h->rhs_stale = false;
    if (mode & 1) {
        h->assembled = true;
        h->matrix_epoch += 1;  // the edge system's values changed (or may have)
    }
    return MH_OK;
}

int read_ctl(mh_handle *h, std::vector<mh::InstCtl> &ctl) {
    ctl.resize(h->sys.n_inst);
    return read_back(h, ctl.data(), h->sys.ctl, sizeof(mh::InstCtl) * ctl.size());
}

// Captures `ipg` CG iterations (two kernels each) into a graph on the handle's own stream;
// with `prof`, an event is recorded after every kernel so each launch can be timed.
int capture_iterations(mh_handle *h, int prec, int ipg, bool prof) {
    const int gi = prec == 64 ? 0 : 1, pi = prof ? 1 : 0;
    if (h->graph[gi][pi] && h->graph_iters[gi][pi] == ipg) return MH_OK;
    if (h->graph[gi][pi]) cudaGraphExecDestroy(h->graph[gi][pi]);
    h->graph[gi][pi] = nullptr;
    if (prof) {
        auto &ev = h->prof_ev[gi];
        while ((int)ev.size() < 2 * ipg + 1) {
            cudaEvent_t e;
            CK(cudaEventCreate(&e));
            ev.push_back(e);
        }
    }
    cudaStream_t cs = h->own_stream;
    cudaGraph_t g;
    CK(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
    cudaError_t e = cudaSuccess;
    // inside a capture only cudaEventRecordExternal turns a record into a graph node
    auto rec = [&](cudaEvent_t ev) { return cudaEventRecordWithFlags(ev, cs, cudaEventRecordExternal); };
    if (prof) e = rec(h->prof_ev[gi][0]);
    for (int k = 0; k < ipg && e == cudaSuccess; ++k) {
        if (prof) {
            e = mh::launch_cg_spmv(h->sys, prec, cs);
            if (e == cudaSuccess) e = rec(h->prof_ev[gi][2 * k + 1]);
            if (e == cudaSuccess) e = mh::launch_cg_update(h->sys, prec, cs);
            if (e == cudaSuccess) e = rec(h->prof_ev[gi][2 * k + 2]);
        } else {
            e = mh::launch_cg_iteration(h->sys, prec, cs);
        }
    }
    cudaError_t e2 = cudaStreamEndCapture(cs, &g);
    if (e != cudaSuccess || e2 != cudaSuccess) {
        if (e2 == cudaSuccess) cudaGraphDestroy(g);
        h->err = cudaGetErrorString(e != cudaSuccess ? e : e2);
        return MH_ERR_CUDA;
    }
    e = cudaGraphInstantiate(&h->graph[gi][pi], g, 0);
    cudaGraphDestroy(g);
    if (e != cudaSuccess) {
        h->graph[gi][pi] = nullptr;
        h->err = cudaGetErrorString(e);
        return MH_ERR_CUDA;
    }
    h->graph_iters[gi][pi] = ipg;
    return MH_OK;
}

// The device-side Krylov loop: a graph of k_loop_init followed by a conditional WHILE node
// whose body is what `body` launches on the capture stream, ending with k_loop_next.  The body
// repeats on the device, with no host round trip, until every instance is done or the body
// count reaches the cap written into d_loop[1] before each launch.
template <class F>
int build_loop_graph(mh_handle *h, F body, cudaGraph_t *out) {
    cudaStream_t cs = h->own_stream;
    cudaGraph_t g = nullptr;
    CK(cudaGraphCreate(&g, 0));
    cudaGraphConditionalHandle hnd{};
    cudaError_t e = cudaGraphConditionalHandleCreate(&hnd, g, 0, 0);
    auto captured = [&](cudaGraph_t target, auto launches) {
        cudaError_t c = cudaStreamBeginCaptureToGraph(cs, target, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
        if (c != cudaSuccess) return c;
        const cudaError_t c1 = launches();
        cudaGraph_t same = nullptr;
        const cudaError_t c2 = cudaStreamEndCapture(cs, &same);
        return c1 != cudaSuccess ? c1 : c2;
    };
    if (e == cudaSuccess) e = captured(g, [&] { return mh::launch_loop_init(h->sys, hnd, h->d_loop, cs); });
    cudaGraphNode_t init = nullptr, loop = nullptr;
    size_t n_nodes = 1;
    if (e == cudaSuccess) e = cudaGraphGetNodes(g, &init, &n_nodes);
    cudaGraphNodeParams cp{};
    cp.type = cudaGraphNodeTypeConditional;
    cp.conditional.handle = hnd;
    cp.conditional.type = cudaGraphCondTypeWhile;
    cp.conditional.size = 1;
    if (e == cudaSuccess) e = cudaGraphAddNode(&loop, g, &init, 1, &cp);
    if (e == cudaSuccess)
        e = captured(cp.conditional.phGraph_out[0], [&] {
            cudaError_t b = body(cs);
            return b != cudaSuccess ? b : mh::launch_loop_next(h->sys, hnd, h->d_loop, cs);
        });
    if (e != cudaSuccess) {
        cudaGraphDestroy(g);
        h->err = std::string("device loop graph: ") + cudaGetErrorString(e);
        cudaGetLastError();
        return MH_ERR_CUDA;
    }
    *out = g;
    return MH_OK;
}

// One launch of a device-loop graph with at most `cap` bodies of `per_body` kernels each; the
// bodies that ran are read back for the launch count.
int run_loop(mh_handle *h, cudaGraphExec_t exec, int64_t cap, int64_t per_body) {
    h->h_done[2] = (int32_t)std::min<int64_t>(std::max<int64_t>(cap, 1), INT32_MAX);
    CK(cudaMemcpyAsync(h->d_loop + 1, h->h_done + 2, sizeof(int32_t), cudaMemcpyHostToDevice, h->stream));
    CK(cudaGraphLaunch(exec, h->stream));
    CK(cudaMemcpyAsync(h->h_done + 3, h->d_loop, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->n_launch += 1 + (int64_t)h->h_done[3] * (per_body + 1);
    return MH_OK;
}

// Krylov iterations in the device-side loop: `ipg` CG iterations per body.
int run_krylov_loop(mh_handle *h, int prec, int ipg, int max_it) {
    const int gi = prec == 64 ? 0 : 1;
    if (!h->loop_graph[gi] || h->loop_iters[gi] != ipg) {
        if (h->loop_graph[gi]) cudaGraphExecDestroy(h->loop_graph[gi]);
        h->loop_graph[gi] = nullptr;
        cudaGraph_t g = nullptr;
        int rc = build_loop_graph(
            h,
            [&](cudaStream_t cs) {
                cudaError_t e = cudaSuccess;
                for (int k = 0; k < ipg && e == cudaSuccess; ++k) e = mh::launch_cg_iteration(h->sys, prec, cs);
                return e;
            },
            &g);
        if (rc) return rc;
        cudaError_t e = cudaGraphInstantiate(&h->loop_graph[gi], g, 0);
        cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            h->loop_graph[gi] = nullptr;
            h->err = cudaGetErrorString(e);
            return MH_ERR_CUDA;
        }
        h->loop_iters[gi] = ipg;
    }
    return run_loop(h, h->loop_graph[gi], ((int64_t)max_it + 2 * ipg) / ipg + 1, 2 * (int64_t)ipg);
}

// The plan of the shared-memory-resident run, made once per handle and precision.  Batches keep
// the two-kernel iteration: its launches are shared by all instances.  A plan whose buffers cannot be had
// leaves nothing behind: no memory, and no error for the next launch to read as its own.
bool resident_ready(mh_handle *h, int prec) {
    const int gi = prec == 64 ? 0 : 1;
    if (h->res_state[gi] == 0) {
        h->res_state[gi] = -1;
        mh::ResidentPlan &pl = h->res_plan[gi];
        mh::ResidentDev &d = h->res_dev[gi];
        if (h->sys.n_inst == 1 && mh::plan_resident(h->hs.slice_off, h->hs.sell_col, h->hs.diag_slot, prec, pl)) {
            const size_t mark = h->allocs.size();
            const std::string err = h->err;
            const size_t np = 16 * (size_t)pl.n_blocks, nq = (prec == 64 ? 4 : 2) * (size_t)h->sys.n_rows;
            d.part = dalloc<double>(h, np);
            d.q = dalloc<double>(h, nq);
            d.err = dalloc<int32_t>(h, 1);
            if (d.part && d.q && d.err && !upload(h, d.blk_slice, pl.blk_slice) &&
                !upload(h, d.halo_off, pl.halo_off) && !upload(h, d.halo_row, pl.halo_row) &&
                !upload(h, d.idx, pl.idx) && !upload(h, d.tag, std::vector<unsigned long long>{1}) &&
                cudaMemsetAsync(d.part, 0, np * sizeof(double), h->stream) == cudaSuccess &&
                cudaMemsetAsync(d.q, 0, nq * sizeof(double), h->stream) == cudaSuccess) {
                h->res_state[gi] = 1;
            } else {
                cudaStreamSynchronize(h->stream);
                for (size_t k = mark; k < h->allocs.size(); ++k) cudaFree(h->allocs[k]);
                h->allocs.resize(mark);
                h->err = err;
                d = mh::ResidentDev();
                cudaGetLastError();
            }
        }
        std::vector<uint16_t>().swap(pl.idx);
    }
    return h->res_state[gi] == 1;
}

// How a Krylov run begins: what its caller has launched before it, once more.
using Restart = std::function<cudaError_t()>;

// The resident run.  done = false: its launch was refused (the chip is shared) or an exchange did not
// complete in its bounded wait.  The run is then back at its start, x as it was, and the handle
// keeps to the two-kernel iteration.  (MH_RESIDENT_POLLS: a shorter wait.)
int run_resident(mh_handle *h, int prec, const Restart &restart, bool &done) {
    const int gi = prec == 64 ? 0 : 1;
    const size_t bytes = (size_t)h->sys.n_rows * sizeof(double);
    int polls = mh::kResidentPolls;
    if (const char *e = getenv("MH_RESIDENT_POLLS")) {
        char *end = nullptr;
        const long v = std::strtol(e, &end, 10);
        if (end != e && v >= 0 && v < polls) polls = (int)v;
    }
    // the FP64 run works on x itself; q is idle in it (the FP32 run leaves x alone)
    if (prec == 64) CK(cudaMemcpyAsync(h->sys.q, h->sys.x, bytes, cudaMemcpyDeviceToDevice, h->stream));
    const cudaError_t e = mh::launch_cg_resident(h->sys, h->res_plan[gi], h->res_dev[gi], polls, h->stream);
    done = e == cudaSuccess;
    if (done) {
        h->n_launch += 1;
        CK(cudaMemcpyAsync(h->h_done, h->res_dev[gi].err, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
        done = *h->h_done == 0;
    }
    if (done) return MH_OK;
    cudaGetLastError();
    h->res_state[gi] = -1;
    if (prec == 64) CK(cudaMemcpyAsync(h->sys.x, h->sys.q, bytes, cudaMemcpyDeviceToDevice, h->stream));
    CK(restart());
    return MH_OK;
}

// Runs captured Krylov iterations until every instance reports done: in the device-side loop,
// or (host_loop, or `prof`) as graphs of `ipg` iterations launched while the host sees an
// instance running.  With `prof`, the kernels of the iterations that still did work are timed
// from the in-graph events.  A system that fits on the chip runs there (with a `restart` to go back to).
int run_krylov(mh_handle *h, int prec, int ipg, int max_it, bool prof, const Restart &restart = nullptr) {
    ipg = std::max(1, ipg);  // an empty graph would never make progress
    if (!prof && !h->host_loop && restart && resident_ready(h, prec)) {
        bool done;
        const int rc = run_resident(h, prec, restart, done);
        if (rc || done) return rc;
    }
    if (!prof && !h->host_loop && !h->loop_unavailable) {
        const int rc = run_krylov_loop(h, prec, ipg, max_it);
        if (rc != MH_ERR_CUDA || h->loop_graph[prec == 64 ? 0 : 1]) return rc;
        h->loop_unavailable = true;  // the loop graph itself failed: the host-polled form
    }
    const int gi = prec == 64 ? 0 : 1, pi = prof ? 1 : 0;
    int rc = capture_iterations(h, prec, ipg, prof);
    if (rc) return rc;
    const int n_inst = h->sys.n_inst;
    int64_t launched = 0;
    std::vector<mh::InstCtl> ctl;
    int it_before = 0;
    if (prof) {
        if ((rc = read_ctl(h, ctl))) return rc;
        for (auto &c : ctl) it_before = std::max(it_before, c.iter);
    }
    while (true) {
        CK(cudaMemcpyAsync(h->h_done, h->sys.n_done, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
        if (*h->h_done >= n_inst) break;
        if (launched > (int64_t)max_it + 2 * ipg) break;  // the device caps iterations itself
        CK(cudaGraphLaunch(h->graph[gi][pi], h->stream));
        launched += ipg;
        h->n_launch += 2 * ipg;
        if (prof) {
            if ((rc = read_ctl(h, ctl))) return rc;
            int it_now = 0;
            for (auto &c : ctl) it_now = std::max(it_now, c.iter);
            const int active = std::min(ipg, it_now - it_before);
            it_before = it_now;
            const int ks = prec == 64 ? MH_KERNEL_SPMV64 : MH_KERNEL_SPMV32;
            for (int k = 0; k < active; ++k) {
                float a = 0.f, b = 0.f;
                CK(cudaEventElapsedTime(&a, h->prof_ev[gi][2 * k], h->prof_ev[gi][2 * k + 1]));
                CK(cudaEventElapsedTime(&b, h->prof_ev[gi][2 * k + 1], h->prof_ev[gi][2 * k + 2]));
                h->kernel_ms[ks] += a;
                h->kernel_ms[ks + 1] += b;
                h->kernel_count[ks] += 1;
                h->kernel_count[ks + 1] += 1;
            }
        }
    }
    return MH_OK;
}

// FP64 true residual per instance: rel = |b - S x| / |b| and abs = |b - S x| (unscaled).
int true_residual(mh_handle *h, std::vector<double> &sums) {
    CK(mh::launch_residual64(h->sys, h->stream));
    h->n_launch += 1;
    sums.resize(mh::kSumStride * (size_t)h->sys.n_inst);
    return read_back(h, sums.data(), h->sys.inst_sums, sizeof(double) * sums.size());
}

struct SolveResult {
    int status = MH_OK;
    int iterations = 0, outer = 0, fell_back = 0;
    double rel = 0.0;       // worst Jacobi-scaled relative true residual
    double rel_orig = 0.0;  // worst unscaled relative true residual
    double ms_setup = 0.0;  // preconditioner setup
};

// Convergence test on the FP64 true residual of every instance: the Jacobi-scaled relative
// residual |D^-1/2 (b - S x)| / |D^-1/2 b| and the unscaled |b - S x| / |b| must both be
// <= r_tol (or the unscaled absolute residual <= a_tol).  Marks unconverged instances
// active in `sums`; returns the worst ratio achieved/target (<= 1 when all converged).
double evaluate(mh_handle *h, const mh_solve_opts &o, std::vector<double> &sums, SolveResult &res, bool &finite) {
    const int n_inst = h->sys.n_inst;
    double worst = 0.0;
    res.rel = res.rel_orig = 0.0;
    finite = true;
    for (int i = 0; i < n_inst; ++i) {
        double *s = &sums[mh::kSumStride * i];
        double rs = std::sqrt(s[0]), bs = std::sqrt(s[3]), ro = std::sqrt(s[1]), bo = std::sqrt(s[2]);
        double rel_s = bs > 0.0 ? rs / bs : 0.0, rel_o = bo > 0.0 ? ro / bo : 0.0;
        if (!std::isfinite(rel_s) || !std::isfinite(rel_o)) finite = false;
        res.rel = std::max(res.rel, rel_s);
        res.rel_orig = std::max(res.rel_orig, rel_o);
        double ratio = (o.r_tol > 0.0) ? std::max(rel_s, rel_o) / o.r_tol : (ro > 0.0 ? 1e300 : 0.0);
        if (ro <= o.a_tol) ratio = 0.0;
        s[mh::kSumActive] = ratio > 1.0 ? 1.0 : 0.0;
        worst = std::max(worst, ratio);
        h->inst_rel[i] = rel_s;
        if (h->inst_status[i] >= 0) h->inst_status[i] = ratio > 1.0 ? MH_NOT_CONVERGED : MH_OK;
    }
    return worst;
}

void count_iterations(mh_handle *h, const std::vector<mh::InstCtl> &ctl) {
    for (size_t i = 0; i < ctl.size(); ++i) {
        h->inst_iters[i] += ctl[i].iter;
        if (ctl[i].status < 0) h->inst_status[i] = ctl[i].status;
    }
}

int solve_pcg64(mh_handle *h, const mh_solve_opts &o, SolveResult &res) {
    std::vector<double> sums;
    std::vector<mh::InstCtl> ctl;
    double tau = o.r_tol;
    int total = 0;
    for (int run = 0; run < 12; ++run) {
        const Restart begin = [&] {
            const cudaError_t e = mh::launch_reset_ctl(h->sys, h->stream);
            h->n_launch += 1;
            return e != cudaSuccess ? e
                                    : mh::launch_cg_init(h->sys, tau * tau, 0.0, std::max(1, o.max_it - total), run > 0,
                                                         h->stream);
        };
        CK(begin());
        int rc = run_krylov(h, 64, o.iters_per_graph, o.max_it - total, o.profile_kernels != 0, begin);
        if (rc) return rc;
        if ((rc = read_ctl(h, ctl))) return rc;
        count_iterations(h, ctl);
        int worst = 0, maxit = 0;
        for (auto &c : ctl) {
            maxit = std::max(maxit, c.iter);
            if (c.status < 0) worst = c.status;
        }
        total += maxit;
        if ((rc = true_residual(h, sums))) return rc;
        bool finite;
        double worst_ratio = evaluate(h, o, sums, res, finite);
        res.outer = run + 1;
        res.iterations = total;
        if (!finite) {
            res.status = MH_ERR_NONFINITE;
            return MH_OK;
        }
        if (worst_ratio <= 1.0) return MH_OK;
        if (worst < 0) {
            res.status = worst;
            return MH_OK;
        }
        if (total >= o.max_it) {
            res.status = MH_NOT_CONVERGED;
            return MH_OK;
        }
        CK(cudaMemcpyAsync(h->sys.inst_sums, sums.data(), sizeof(double) * sums.size(), cudaMemcpyHostToDevice,
                           h->stream));
        tau = tau / (2.0 * worst_ratio);
        if (tau < 1e-300) tau = 1e-300;
    }
    res.status = MH_NOT_CONVERGED;
    return MH_OK;
}

// Mixed precision: the Krylov recursion runs in FP32 (SpMV with FP32 values, FP32 vectors,
// FP64 dot products) while x and the true residual are kept in FP64.  Whenever the FP32
// residual has dropped by inner_rtol (or inner_max_it iterations have passed), the FP32
// correction is folded into x64, r64 = b - S x64 is recomputed in FP64, and the recursion
// continues from r64 with the same search direction (reliable update).  If the FP64
// residual stops decreasing, the solve finishes with FP64 PCG from the current x.
int solve_ir32(mh_handle *h, const mh_solve_opts &o, SolveResult &res) {
    std::vector<double> sums;
    std::vector<mh::InstCtl> ctl;
    int total = 0;
    double best = 1e300;
    int stall = 0;
    for (int outer = 0; outer < 1000; ++outer) {
        int rc = true_residual(h, sums);
        if (rc) return rc;
        bool finite;
        double worst_ratio = evaluate(h, o, sums, res, finite);
        if (!finite) {
            res.status = MH_ERR_NONFINITE;
            return MH_OK;
        }
        res.outer = outer;
        res.iterations = total;
        if (worst_ratio <= 1.0) return MH_OK;
        if (total >= o.max_it) {
            res.status = MH_NOT_CONVERGED;
            return MH_OK;
        }
        if (worst_ratio < 0.9 * best) {
            best = worst_ratio;
            stall = 0;
        } else if (++stall >= 3) {
            // FP32 recursion stagnates (e.g. conditioning beyond single precision): finish in FP64
            mh_solve_opts o64 = o;
            o64.max_it = std::max(1, o.max_it - total);
            SolveResult r64;
            rc = solve_pcg64(h, o64, r64);
            res.status = r64.status;
            res.rel = r64.rel;
            res.rel_orig = r64.rel_orig;
            res.iterations = total + r64.iterations;
            res.outer = outer + r64.outer;
            res.fell_back = 1;
            return rc;
        }
        CK(cudaMemcpyAsync(h->sys.inst_sums, sums.data(), sizeof(double) * sums.size(), cudaMemcpyHostToDevice,
                           h->stream));
        CK(mh::launch_reset_ctl(h->sys, h->stream));
        const int seg_max = std::min(o.inner_max_it, o.max_it - total);
        if (outer == 0)
            CK(mh::launch_ir_start(h->sys, o.inner_rtol * o.inner_rtol, seg_max, h->stream));
        else
            CK(mh::launch_ir_replace(h->sys, o.inner_rtol * o.inner_rtol, seg_max, h->stream));
        // (a failed resident run has spoilt the direction: a new sequence)
        const Restart again = [&] {
            const cudaError_t e = mh::launch_reset_ctl(h->sys, h->stream);
            return e != cudaSuccess ? e
                                    : mh::launch_ir_start(h->sys, o.inner_rtol * o.inner_rtol, seg_max, h->stream);
        };
        if ((rc = run_krylov(h, 32, o.iters_per_graph, seg_max, o.profile_kernels != 0, again))) return rc;
        CK(mh::launch_ir_correct(h->sys, h->stream));
        h->n_launch += 2;
        if ((rc = read_ctl(h, ctl))) return rc;
        count_iterations(h, ctl);
        int maxit = 0;
        for (auto &c : ctl) maxit = std::max(maxit, c.iter);
        total += maxit;
    }
    res.status = MH_NOT_CONVERGED;
    return MH_OK;
}

// ---- learned preconditioner and flexible CG ----------------------------------------------

// Initial parameters of the smoother network: Xavier-scaled random layers (fixed seed) and a
// zero output layer, so that every weight is 1 (plain smoothing) until training.
void nn_initial_params(std::vector<float> &w, uint64_t seed) {
    w.assign(mh::kSnParams, 0.f);
    std::mt19937_64 rng(seed);
    std::normal_distribution<double> nd(0.0, 1.0);
    const double s0 = std::sqrt(2.0 / (mh::kSnF + mh::kSnW)), s1 = 0.5 * std::sqrt(2.0 / (3 * mh::kSnW));
    for (int k = 0; k < mh::kSnW * mh::kSnF; ++k) w[mh::kSnOffW0 + k] = (float)(s0 * nd(rng));
    for (int l = 0; l < mh::kSnL; ++l)
        for (int k = 0; k < mh::kSnW * 2 * mh::kSnW; ++k) w[mh::kSnOffLayer + l * mh::kSnPerLayer + k] = (float)(s1 * nd(rng));
}

int nn_upload_weights(mh_handle *h, const float *w_host) {
    CK(cudaMemcpyAsync(h->nn_w, w_host, mh::kSnParams * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemsetAsync(h->nn_m, 0, mh::kSnParams * sizeof(float), h->stream));
    CK(cudaMemsetAsync(h->nn_v, 0, mh::kSnParams * sizeof(float), h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->nn_step = 0;
    return MH_OK;
}

int ensure_learned(mh_handle *h) {
    if (h->nn_w) return MH_OK;
    const int64_t nr = h->sys.n_rows;
    h->nn_w = dalloc<float>(h, mh::kSnParams);
    h->nn_m = dalloc<float>(h, mh::kSnParams);
    h->nn_v = dalloc<float>(h, mh::kSnParams);
    h->nn_grad = dalloc<float>(h, mh::kSnParams);
    h->cheb_z0 = dalloc<float>(h, nr);
    h->cheb_z1 = dalloc<float>(h, nr);
    h->cheb_d = dalloc<float>(h, nr);
    h->spec_bound = dalloc<unsigned int>(h, 1);
    h->d_loss = dalloc<double>(h, 1);
    if (!h->nn_w || !h->nn_m || !h->nn_v || !h->nn_grad || !h->cheb_z0 || !h->cheb_z1 || !h->cheb_d ||
        !h->spec_bound || !h->d_loss)
        return MH_ERR_NOMEM;
    std::vector<float> w;
    nn_initial_params(w, 1);
    return nn_upload_weights(h, w.data());
}

// The network's smoother weights for the current matrix into h->sn_w (features recomputed when
// the matrix changed).  The inference buffers are allocated on first use.
int nn_weights(mh_handle *h) {
    int rc;
    if ((rc = ensure_learned(h))) return rc;
    const int64_t nr = h->sys.n_rows;
    if (!h->sn_x) {
        h->sn_x = dalloc<float>(h, nr * mh::kSnF);
        h->sn_w = dalloc<float>(h, nr);
        h->sn_inf.h[0] = dalloc<float>(h, nr * mh::kSnW);
        h->sn_inf.h[1] = dalloc<float>(h, nr * mh::kSnW);
        h->sn_inf.a[0] = dalloc<float>(h, nr * mh::kSnW);
        if (!h->sn_x || !h->sn_w || !h->sn_inf.h[0] || !h->sn_inf.h[1] || !h->sn_inf.a[0]) return MH_ERR_NOMEM;
    }
    if (h->sn_x_epoch != h->matrix_epoch) {
        CK(mh::sn_features(h->sys, h->sn_x, h->stream));
        h->sn_x_epoch = h->matrix_epoch;
        h->n_launch += 1;
    }
    CK(mh::sn_forward(h->sys, h->nn_w, h->sn_x, h->sn_inf, h->sn_w, false, h->stream));
    h->n_launch += 2 + 2 * mh::kSnL;
    return MH_OK;
}

// Upper bound of the spectrum of the scaled FP32 system (Gershgorin).
int spectrum_bound(mh_handle *h, double &hi) {
    CK(mh::launch_spectrum_bound(h->sys, h->spec_bound, h->stream));
    unsigned int bits = 0;
    if (int rc = read_back(h, &bits, h->spec_bound, sizeof(bits))) return rc;
    float f;
    std::memcpy(&f, &bits, sizeof(f));
    hi = f > 0.f ? (double)f : 2.0;
    return MH_OK;
}

// One flexible-CG iteration: z = M(r) (network, Chebyshev polynomial or AMG V-cycle) with
// beta = z.q_old / (p.q)_old, p = z - beta p, q = S^ p with alpha = p.r / p.q, x and r.
cudaError_t fcg_iteration(mh_handle *h, Pc kind, int degree, double lo, double hi, cudaStream_t s,
                          mh::AmgProf *prof = nullptr, bool follows = false) {
    mh::DevSystem &sys = h->sys;
    cudaError_t e;
    switch (kind) {
        case Pc::Cheb:
            e = mh::launch_cheb_apply(sys, sys.r32, h->cheb_z0, h->cheb_z1, h->cheb_d, sys.z32, degree, lo, hi, s,
                                      follows);
            break;
        default:
            e = h->amg.apply(sys.r32, sys.z32, sys.n_done, sys.n_inst, s, prof, follows);
            break;
    }
    return e == cudaSuccess ? mh::launch_fcg_iteration(sys, sys.z32, s, !prof) : e;
}

int fcg_kernels_per_iteration(mh_handle *h, Pc kind, int degree) {
    switch (kind) {
        case Pc::Cheb: return degree + 2;
        default: return h->amg.kernels_per_apply() + 2;
    }
}

void drop_fcg_graph(mh_handle *h) {
    if (h->fcg_graph) cudaGraphExecDestroy(h->fcg_graph);
    h->fcg_graph = nullptr;
}

// Runs captured FCG iterations until every instance reports done.  The graph is kept while
// its inputs (preconditioner, launch shape, AMG hierarchy) stay the same.
// With prof (AMG only), every V-cycle of the graph records timing events; the cycles of the
// iterations that did work are added to the MH_KERNEL_VCYCLE / MH_KERNEL_SMOOTH0 classes.
int run_fcg(mh_handle *h, Pc kind, int degree, double lo, double hi, int ipg, int max_it, bool prof) {
    ipg = std::max(1, ipg);  // an empty graph would never make progress
    prof = prof && (kind == Pc::Amg || kind == Pc::Nn);
    const bool loop = !prof && !h->host_loop && !h->loop_unavailable;
    const FcgKey key{(int)kind, ipg, degree, lo, hi, h->amg_epoch, prof, loop};
    if (prof) {
        const int steps = h->amg.fine_steps();
        if ((int)h->amg_prof.size() < ipg) h->amg_prof.resize(ipg);
        for (auto &p : h->amg_prof) {
            for (auto &e : p.cycle)
                if (!e) CK(cudaEventCreate(&e));
            while ((int)p.smooth.size() < 2 * steps) {
                cudaEvent_t e;
                CK(cudaEventCreate(&e));
                p.smooth.push_back(e);
            }
        }
    }
    if (!h->fcg_graph || !(h->fcg_key == key)) {
        cudaGraph_t g;
        cudaError_t e = cudaSuccess;
        if (loop) {
            const int rc = build_loop_graph(
                h,
                [&](cudaStream_t cs) {
                    cudaError_t b = cudaSuccess;
                    for (int k = 0; k < ipg && b == cudaSuccess; ++k)
                        b = fcg_iteration(h, kind, degree, lo, hi, cs, nullptr, k > 0);
                    return b;
                },
                &g);
            if (rc) {  // the loop graph itself failed: the host-polled form from now on
                h->loop_unavailable = true;
                return run_fcg(h, kind, degree, lo, hi, ipg, max_it, prof);
            }
        } else {
            CK(cudaStreamBeginCapture(h->own_stream, cudaStreamCaptureModeThreadLocal));
            for (int k = 0; k < ipg && e == cudaSuccess; ++k)
                e = fcg_iteration(h, kind, degree, lo, hi, h->own_stream, prof ? &h->amg_prof[k] : nullptr, k > 0);
            cudaError_t e2 = cudaStreamEndCapture(h->own_stream, &g);
            if (e != cudaSuccess || e2 != cudaSuccess) {
                if (e2 == cudaSuccess) cudaGraphDestroy(g);
                h->err = cudaGetErrorString(e != cudaSuccess ? e : e2);
                cudaGetLastError();
                return MH_ERR_CUDA;
            }
        }
        // a new hierarchy of the same shape (the usual case when only values changed) only
        // changes kernel parameters: update the executable graph in place
        bool updated = false;
        if (h->fcg_graph && h->fcg_key.kind == key.kind && h->fcg_key.ipg == key.ipg && h->fcg_key.prof == prof &&
            h->fcg_key.loop == loop) {
            cudaGraphExecUpdateResultInfo info;
            updated = cudaGraphExecUpdate(h->fcg_graph, g, &info) == cudaSuccess;
            if (!updated) cudaGetLastError();
        }
        if (!updated) {
            drop_fcg_graph(h);
            e = cudaGraphInstantiate(&h->fcg_graph, g, 0);
        }
        cudaGraphDestroy(g);
        if (e != cudaSuccess) {
            h->fcg_graph = nullptr;
            h->err = cudaGetErrorString(e);
            return MH_ERR_CUDA;
        }
        h->fcg_key = key;
    }
    const int per_iter = fcg_kernels_per_iteration(h, kind, degree);
    if (loop) return run_loop(h, h->fcg_graph, ((int64_t)max_it + 2 * ipg) / ipg + 1, (int64_t)per_iter * ipg);
    int64_t launched = 0;
    std::vector<mh::InstCtl> ctl;
    int it_before = 0;
    if (prof) {
        int rc = read_ctl(h, ctl);
        if (rc) return rc;
        for (auto &c : ctl) it_before = std::max(it_before, c.iter);
    }
    while (true) {
        CK(cudaMemcpyAsync(h->h_done, h->sys.n_done, sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
        if (*h->h_done >= h->sys.n_inst) break;
        if (launched > (int64_t)max_it + 2 * ipg) break;
        CK(cudaGraphLaunch(h->fcg_graph, h->stream));
        launched += ipg;
        h->n_launch += (int64_t)per_iter * ipg;
        if (prof) {
            int rc = read_ctl(h, ctl);
            if (rc) return rc;
            int it_now = 0;
            for (auto &c : ctl) it_now = std::max(it_now, c.iter);
            const int active = std::min(ipg, it_now - it_before);
            it_before = it_now;
            for (int k = 0; k < active; ++k) {
                const mh::AmgProf &p = h->amg_prof[k];
                float ms = 0.f;
                CK(cudaEventElapsedTime(&ms, p.cycle[0], p.cycle[1]));
                h->kernel_ms[MH_KERNEL_VCYCLE] += ms;
                h->kernel_count[MH_KERNEL_VCYCLE] += 1;
                for (int q = 0; q + 1 < 2 * h->amg.fine_steps() && q + 1 < (int)p.smooth.size(); q += 2) {
                    CK(cudaEventElapsedTime(&ms, p.smooth[q], p.smooth[q + 1]));
                    h->kernel_ms[MH_KERNEL_SMOOTH0] += ms;
                    h->kernel_count[MH_KERNEL_SMOOTH0] += 1;
                }
            }
        }
    }
    return MH_OK;
}

// AMG options: defaults, overridable from the environment for tuning studies
mh::AmgOptions amg_options() {
    mh::AmgOptions o;
    auto env_i = [](const char *k, int &v, int lo, int hi) {
        if (const char *e = getenv(k)) {
            const int x = atoi(e);
            if (x >= lo && x <= hi) v = x;
        }
    };
    env_i("MH_AMG_DEGREE", o.cheb_degree, 1, 8);
    env_i("MH_AMG_PRE", o.pre_degree, 0, 8);
    env_i("MH_AMG_PASSES", o.pair_passes, 1, 4);
    env_i("MH_AMG_CPASSES", o.pair_passes_coarse, 1, 4);
    env_i("MH_AMG_COARSE", o.coarse_max, 16, 1280);
    env_i("MH_AMG_ROUNDS", o.pair_rounds, 1, 16);
    env_i("MH_AMG_KCYCLE", o.kcycle, 0, 1);
    env_i("MH_AMG_KLEVELS", o.kcycle_levels, 0, 64);
    env_i("MH_AMG_WEIGHTED", o.weighted, 0, 1);
    env_i("MH_AMG_MIX", o.mix_coarse, 0, 1);
    env_i("MH_AMG_SPLIT", o.split, 0, 8);
    env_i("MH_AMG_SPLITW", o.split_width, 2, 64);
    env_i("MH_AMG_HALF", o.half_fine, 0, 1);
    if (const char *e = getenv("MH_AMG_RATIO")) {
        const float x = (float)atof(e);
        if (x >= 1.5f && x <= 100.f) o.cheb_ratio = x;
    }
    if (const char *e = getenv("MH_AMG_ALPHA")) {
        const float x = (float)atof(e);
        if (x > 0.f && x <= 3.f) o.alpha = x;
    }
    env_i("MH_AMG_POWER", o.power_steps, 0, 64);
    env_i("MH_AMG_TAIL", o.tail_rows, 0, 1 << 22);
    env_i("MH_AMG_LEVELS", o.max_levels, 2, 20);
    env_i("MH_AMG_CDEG", o.coarse_degree, 1, 64);
    env_i("MH_AMG_TMA", o.fine_tma, 0, 1);
    env_i("MH_AMG_TMA_STAGES", o.fine_tma_stages, 2, 4);
    env_i("MH_AMG_STALL", o.stall_rows, 0, 1 << 24);
    if (const char *e = getenv("MH_AMG_CRATIO")) {
        const float x = (float)atof(e);
        if (x >= 2.f && x <= 1000.f) o.coarse_ratio = x;
    }
    if (const char *e = getenv("MH_AMG_SAFETY")) {
        const float x = (float)atof(e);
        if (x >= 1.f && x <= 3.f) o.power_safety = x;
    }
    return o;
}

// the options with what mh_autotune_ex chose for this handle
mh::AmgOptions amg_options_for(const mh_handle *h) {
    mh::AmgOptions o = amg_options();
    if (h->amg_fine_passes > 0) o.pair_passes = h->amg_fine_passes;
    return o;
}


// The multigrid preconditioner for the current matrix, with the fine level's smoother weights
// of the method: the network's (learned method), the caller's (mh_smoother_weights_set), or
// none.  The hierarchy is rebuilt when the matrix changed (ms_setup: its device time, else 0);
// MH_FELL_BACK when the setup failed (h->err says why).
int prepare_multigrid(mh_handle *h, Pc kind, double &ms_setup) {
    int rc;
    ms_setup = 0.0;
    // the fine level's smoother weights: the network's (learned method), the caller's
    // (mh_smoother_weights_set), or none
    const float *want = nullptr;
    if (kind == Pc::Nn) {
        if (h->sn_key_epoch != h->matrix_epoch || h->sn_key_step != h->nn_step || !h->sn_w) {
            if ((rc = nn_weights(h))) return rc;
            h->sn_key_epoch = h->matrix_epoch;
            h->sn_key_step = h->nn_step;
            h->amg.set_fine_weights(nullptr);  // new values: the interval is re-estimated below
        }
        want = h->sn_w;
    } else if (h->user_fine_w) {
        want = h->d_fine_w;
    }
    if (h->amg_matrix_epoch == h->matrix_epoch && h->amg.levels() > 0) {
        // same matrix as the hierarchy was built from (unsteady steps at a fixed dt): the
        // hierarchy is reused, with the fine interval re-estimated when the weights changed
        ms_setup = 0.0;
        if (h->amg.fine_smoother_weights() != want) {
            h->amg.set_fine_weights(want);
            CK(h->amg.refresh_fine(h->stream));
            h->amg_epoch += 1;  // captured cycles hold the old smoothing coefficients
        }
    } else {
        // the hierarchy is built from the current matrix values
        h->amg.set_fine_weights(want);
        h->amg_training = false;
        h->amg_epoch += 1;
        h->amg_matrix_epoch = h->matrix_epoch;
        CK(cudaEventRecord(h->ev[6], h->stream));
        cudaError_t e = h->amg.setup(h->sys, amg_options_for(h), h->stream);
        CK(cudaEventRecord(h->ev[7], h->stream));
        CK(cudaEventSynchronize(h->ev[7]));
        float ms = 0.f;
        CK(cudaEventElapsedTime(&ms, h->ev[6], h->ev[7]));
        ms_setup = ms;
        h->n_launch += h->amg.levels() * 12;
        if (e != cudaSuccess) {
            h->err = "AMG setup: " + h->amg.err;
            cudaGetLastError();
            h->amg_matrix_epoch = -1;
            return MH_FELL_BACK;
        }
    }
    return MH_OK;
}

// Mixed-precision flexible CG: FP32 FCG with the multigrid (plain or with the learned smoother)
// or Chebyshev-Jacobi preconditioner inside FP64 reliable updates, as solve_ir32; the direction
// sequence runs on across them.  If a segment of the learned method breaks down, uses up
// inner_max_it, or the FP64 residual stops improving over three replacements, Chebyshev-Jacobi
// replaces it for the rest of the solve (fell_back = 1), with segments of at least
// kFallbackSegment iterations.
constexpr int kFallbackSegment = 200;

// One FP32 segment: flexible CG on S^ d = r / |r| for the instances that `sums` marks active, until
// the residual is down by `rtol`, and x += |r| d.  fresh: a new direction sequence.
int fcg_segment(mh_handle *h, const mh_solve_opts &o, Pc kind, int degree, double hi, const std::vector<double> &sums,
                double rtol, int seg_max, bool fresh, std::vector<mh::InstCtl> &ctl) {
    CK(cudaMemcpyAsync(h->sys.inst_sums, sums.data(), sizeof(double) * sums.size(), cudaMemcpyHostToDevice, h->stream));
    CK(mh::launch_reset_ctl(h->sys, h->stream));
    if (fresh)
        CK(mh::launch_ir_start(h->sys, rtol * rtol, seg_max, h->stream));
    else
        CK(mh::launch_ir_continue(h->sys, rtol * rtol, seg_max, h->stream));
    int rc = run_fcg(h, kind, degree, hi / 30.0, hi, o.iters_per_graph, seg_max, o.profile_kernels != 0);
    if (rc) return rc;
    CK(mh::launch_ir_correct(h->sys, h->stream));
    h->n_launch += 2;
    return read_ctl(h, ctl);
}

int most_iterations(const std::vector<mh::InstCtl> &ctl) {
    int most = 0;
    for (auto &c : ctl) most = std::max(most, c.iter);
    return most;
}

// A tolerance of the order of the FP64 rounding asks for the pressures as exactly as they come; side
// fluxes are differences of them and lose three to four more decimals.  A multigrid segment lowers the
// residual by about 1e-3, so a solve to 1e-15 ends anywhere between r_tol and a hundredth of it, far
// above what FP64 can reach (1e-18 of the right-hand side on 3.2M edges): flux vectors were off by 6e-8
// (largest difference over the RMS) where it ended at 0.3-0.46 r_tol, and by 1e-8 at most below 0.1.
// Such a solve ends a decimal below r_tol: an instance above that gets one more short segment, which
// is undone if it does not lower the residual (FP64 rounding reached first).
constexpr double kRoundingTol = 8.0 * std::numeric_limits<double>::epsilon();
constexpr double kRoundingShare = 0.1;

int polish(mh_handle *h, const mh_solve_opts &o, SolveResult &res, Pc kind, int degree, double hi,
           std::vector<double> &sums, double worst) {
    const int seg_max = std::min(o.inner_max_it, o.max_it - res.iterations);
    const size_t bytes = (size_t)h->sys.n_rows * sizeof(double);
    if (seg_max <= 0) return MH_OK;
    if (!h->x_keep && !(h->x_keep = dalloc<double>(h, h->sys.n_rows))) {
        cudaGetLastError();
        return MH_OK;
    }
    const std::vector<int32_t> status = h->inst_status;
    const std::vector<double> rel = h->inst_rel;
    const SolveResult before = res;
    mh_solve_opts tight = o;
    tight.r_tol *= kRoundingShare;
    bool finite;
    evaluate(h, tight, sums, res, finite);  // marks the instances above
    CK(cudaMemcpyAsync(h->x_keep, h->sys.x, bytes, cudaMemcpyDeviceToDevice, h->stream));
    std::vector<mh::InstCtl> ctl;
    int rc = fcg_segment(h, o, kind, degree, hi, sums, kRoundingShare, seg_max, false, ctl);
    if (rc || (rc = true_residual(h, sums))) return rc;
    for (size_t i = 0; i < ctl.size(); ++i) h->inst_iters[i] += ctl[i].iter;
    h->inst_status = status;
    const double now = evaluate(h, o, sums, res, finite);
    if (!finite || !(now < worst)) {
        CK(cudaMemcpyAsync(h->sys.x, h->x_keep, bytes, cudaMemcpyDeviceToDevice, h->stream));
        h->inst_status = status;
        h->inst_rel = rel;
        res = before;
    }
    res.iterations = before.iterations + most_iterations(ctl);
    res.outer = before.outer + 1;
    return MH_OK;
}

int solve_fcg(mh_handle *h, const mh_solve_opts &o, SolveResult &res, Pc kind) {
    int rc = ensure_learned(h);
    if (rc) return rc;
    if (h->sys.rows_per_thread != 1) {  // the preconditioner kernels work on tiles of 256 rows
        const int t[2] = {mh::krylov_target_blocks(1, 64), mh::krylov_target_blocks(1, 32)};
        if ((rc = apply_launch_shape(h, 1, t))) return rc;
    }
    double hi = 0.0;  // spectrum bound of the Chebyshev-Jacobi polynomial, once that is used
    const int degree = std::max(1, std::min(o.cheb_degree, 16));
    if (kind == Pc::Amg || kind == Pc::Nn) {
        if ((rc = prepare_multigrid(h, kind, res.ms_setup))) {
            if (rc != MH_FELL_BACK) return rc;
            kind = Pc::Cheb;  // the polynomial preconditioner needs no setup
            res.fell_back = 1;
        }
    }
    std::vector<double> sums;
    std::vector<mh::InstCtl> ctl;
    int total = 0, stall = 0;
    double best = 1e300;
    const bool learned = kind == Pc::Nn;
    bool use_nn = learned, restart = false;
    for (int outer = 0; outer < 1000; ++outer) {
        if ((rc = true_residual(h, sums))) return rc;
        bool finite;
        double worst_ratio = evaluate(h, o, sums, res, finite);
        if (!finite) {
            res.status = MH_ERR_NONFINITE;
            return MH_OK;
        }
        res.outer = outer;
        res.iterations = total;
        if (worst_ratio <= 1.0) {
            const bool multigrid = learned ? use_nn : kind == Pc::Amg;
            if (outer > 0 && multigrid && o.r_tol <= kRoundingTol && worst_ratio > kRoundingShare)
                return polish(h, o, res, kind, degree, hi, sums, worst_ratio);
            return MH_OK;
        }
        if (total >= o.max_it) {
            res.status = MH_NOT_CONVERGED;
            return MH_OK;
        }
        if (worst_ratio < 0.9 * best) {
            best = worst_ratio;
            stall = 0;
        } else if (++stall >= 3) {
            if (use_nn) {
                use_nn = false;
                res.fell_back = 1;
                stall = 0;
                best = 1e300;
                restart = true;
                std::fill(h->inst_status.begin(), h->inst_status.end(), 0);
            } else {
                res.status = MH_NOT_CONVERGED;
                return MH_OK;
            }
        }
        // a fallback gets segments long enough to make progress whatever limit the learned
        // method was given
        const int seg_lim = learned && !use_nn ? std::max(o.inner_max_it, kFallbackSegment) : o.inner_max_it;
        const int seg_max = std::min(seg_lim, o.max_it - total);
        const Pc cur = learned ? (use_nn ? Pc::Nn : Pc::Cheb) : kind;
        if (cur == Pc::Cheb && hi == 0.0 && (rc = spectrum_bound(h, hi))) return rc;
        // the direction sequence continues across replacements unless the preconditioner changed
        if ((rc = fcg_segment(h, o, cur, degree, hi, sums, o.inner_rtol, seg_max, outer == 0 || restart, ctl))) return rc;
        restart = false;
        count_iterations(h, ctl);
        bool seg_bad = false;  // an instance broke down or used up the segment's iterations
        for (auto &c : ctl)
            if (c.status != 0) seg_bad = true;
        total += most_iterations(ctl);
        if (seg_bad && use_nn) {
            use_nn = false;
            res.fell_back = 1;
            stall = 0;
            restart = true;
            std::fill(h->inst_status.begin(), h->inst_status.end(), 0);  // the fallback takes over
        }
    }
    res.status = MH_NOT_CONVERGED;
    return MH_OK;
}

int ensure_train(mh_handle *h, int n_pairs) {
    const int64_t nr = h->sys.n_rows;
    if (!h->tr_ready) {
        const size_t big = (size_t)nr * mh::kSnW;
        bool ok = true;
        for (auto &v : h->sn_tr.h) ok &= (v = dalloc<float>(h, big)) != nullptr;
        for (auto &v : h->sn_tr.a) ok &= (v = dalloc<float>(h, big)) != nullptr;
        for (auto &v : h->sn_tr.u) ok &= (v = dalloc<float>(h, big)) != nullptr;
        ok &= (h->sn_tr.u0 = dalloc<float>(h, big)) != nullptr;
        ok &= (h->sn_tr.z = dalloc<float>(h, nr)) != nullptr;
        ok &= (h->sn_sc.dz = dalloc<float>(h, nr)) != nullptr;
        ok &= (h->sn_sc.dh = dalloc<float>(h, big)) != nullptr;
        ok &= (h->sn_sc.du = dalloc<float>(h, big)) != nullptr;
        ok &= (h->sn_sc.da = dalloc<float>(h, big)) != nullptr;
        ok &= (h->sn_sc.part = dalloc<float>(h, (size_t)mh::kSnWgradBlocks * (mh::kSnW * 2 * mh::kSnW + mh::kSnW))) !=
              nullptr;
        for (auto &v : h->tv) ok &= (v = dalloc<float>(h, nr)) != nullptr;
        ok &= (h->tdot = dalloc<double>(h, 256)) != nullptr;
        ok &= (h->pair_acc = dalloc<double>(h, 2)) != nullptr;
        if (!ok) return MH_ERR_NOMEM;
        h->tr_ready = true;
    }
    if (h->pair_cap < n_pairs) {
        h->pair_r = dalloc<float>(h, (size_t)n_pairs * nr);
        h->pair_e = dalloc<float>(h, (size_t)n_pairs * nr);
        if (!h->pair_r || !h->pair_e) return MH_ERR_NOMEM;
        h->pair_cap = n_pairs;
    }
    return MH_OK;
}

// Multigrid options of training: the cycle without the energy-optimal coarse scaling (so that
// it is linear in the residual and its adjoint exact) and with FP32 fine values (those of the
// adjoint's products)
mh::AmgOptions training_amg_options(const mh_handle *h) {
    mh::AmgOptions o = amg_options_for(h);
    o.kcycle = 0;
    o.half_fine = 0;
    return o;
}

// One training evaluation on pair k (r, e in the solver rows, e'S^e = er): the network gives the
// smoother weights w; M is the V-cycle with them; the loss is L = (x3 - e)' S^ (x3 - e) / er for
// x3 = M r, and dw = dL/dw comes from the cycle's adjoint.  With the cycle
//   x1 = Q r,  x2 = x1 + P B P' (r - S^ x1),  x3 = x2 + Q (r - S^ x2),   Q = a0 W + a1 W S^ W,
// g = 2 S^ (x3 - e) / er, u = g - S^ Q g, hh = u - S^ P B P' u and r2 = r - S^ x2:
//   dL/dw_i = a0 (g_i r2_i + hh_i r_i) + a1 (g_i (S^W r2)_i + (S^W g)_i r2_i + hh_i (S^W r)_i
//             + (S^W hh)_i r_i)
// (the smoothing interval is held fixed: refresh = 1 re-estimates it for the current weights
// first).  Then grad = dL/dtheta through the network's backward kernels.  The loss goes to *loss
// (host).  The hierarchy must be the training one (training_amg_options) of this matrix.
int train_eval(mh_handle *h, const float *r, const float *e, double er, bool refresh, double *loss) {
    const int64_t nr = h->sys.n_rows;
    mh::DevSystem &S = h->sys;
    cudaStream_t st = h->stream;
    if (h->sn_x_epoch != h->matrix_epoch) {
        CK(mh::sn_features(S, h->sn_x, st));
        h->sn_x_epoch = h->matrix_epoch;
    }
    CK(mh::sn_forward(S, h->nn_w, h->sn_x, h->sn_tr, h->sn_w, true, st));
    h->amg.set_fine_weights(h->sn_w);
    if (refresh) CK(h->amg.refresh_fine(st));
    else CK(h->amg.update_fine_weights(st));
    double a0, a1;
    if (!h->amg.fine_poly(a0, a1)) {
        h->err = "training needs the degree-2 fine smoother";
        return MH_ERR_STATE;
    }
    float **v = h->tv;
    float *x1 = v[0], *t1 = v[1], *r1 = v[2], *c = v[3], *x2 = v[4], *r2 = v[5], *x3 = v[6], *d = v[7];
    float *sd = v[8], *g = v[9], *qg = v[10], *u = v[11], *cu = v[12], *hh = v[13], *swr = v[14], *dw = v[15];
    CK(h->amg.smooth_fine(r, x1, st));
    CK(mh::sn_spmv(S, nullptr, x1, t1, st));
    CK(mh::sn_axpy(nr, r, -1.f, t1, r1, st));
    CK(h->amg.coarse_correct(r1, c, st));
    CK(mh::sn_axpy(nr, x1, 1.f, c, x2, st));
    CK(mh::sn_spmv(S, nullptr, x2, t1, st));
    CK(mh::sn_axpy(nr, r, -1.f, t1, r2, st));
    CK(h->amg.smooth_fine(r2, t1, st));
    CK(mh::sn_axpy(nr, x2, 1.f, t1, x3, st));
    CK(mh::sn_axpy(nr, x3, -1.f, e, d, st));
    CK(mh::sn_spmv(S, nullptr, d, sd, st));
    CK(mh::sn_dot(nr, d, sd, h->tdot, h->tdot + 200, st));
    CK(mh::sn_axpy(nr, sd, (float)(2.0 / er) - 1.f, sd, g, st));
    CK(h->amg.smooth_fine(g, qg, st));
    CK(mh::sn_spmv(S, nullptr, qg, t1, st));
    CK(mh::sn_axpy(nr, g, -1.f, t1, u, st));
    CK(h->amg.coarse_correct(u, cu, st));
    CK(mh::sn_spmv(S, nullptr, cu, t1, st));
    CK(mh::sn_axpy(nr, u, -1.f, t1, hh, st));
    // the four products S^ W v (x1, c and t1 are free again)
    CK(mh::sn_spmv(S, h->amg.fine_smoother_weights_in_effect(), r, swr, st));
    CK(mh::sn_spmv(S, h->amg.fine_smoother_weights_in_effect(), r2, t1, st));
    CK(mh::sn_spmv(S, h->amg.fine_smoother_weights_in_effect(), g, x1, st));
    CK(mh::sn_spmv(S, h->amg.fine_smoother_weights_in_effect(), hh, c, st));
    CK(cudaMemsetAsync(dw, 0, nr * sizeof(float), st));
    const int32_t *agg = h->amg.levels() > 1 ? h->amg.level(0).agg.p : nullptr;
    CK(mh::sn_grad_w(S, (float)a0, (float)a1, g, hh, r, r2, swr, t1, x1, c, agg, 1.f, dw, st));
    CK(mh::sn_backward(S, h->nn_w, h->sn_x, h->sn_tr, dw, h->nn_grad, h->sn_sc, st));
    h->n_launch += 40 + 2 * h->amg.levels() * 8;
    double num = 0.0;
    CK(cudaMemcpyAsync(&num, h->tdot + 200, sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (loss) *loss = num / er;
    return std::isfinite(num) ? MH_OK : MH_ERR_NONFINITE;
}

// Training pairs from the plain solver (FP64 PCG): x* to solve_rtol, then snapshots x_s of a
// rerun from zero at geometrically spaced iterations; pair s = (r_s, e_s = x* - x_s) scaled by
// 1/|r_s|, stored in pair_r / pair_e; er[s] = e_s'r_s after scaling.
int make_pairs(mh_handle *h, int np, double solve_rtol, std::vector<double> &er) {
    int rc;
    const int64_t nr = h->sys.n_rows;
    if (!h->x_star && !(h->x_star = dalloc<double>(h, nr))) return MH_ERR_NOMEM;
    mh_solve_opts so;
    mh_solve_opts_default(&so);
    so.r_tol = solve_rtol > 0.0 ? solve_rtol : 1e-9;
    so.iters_per_graph = 16;
    std::fill(h->inst_iters.begin(), h->inst_iters.end(), 0);
    std::fill(h->inst_status.begin(), h->inst_status.end(), 0);
    CK(cudaMemsetAsync(h->sys.x, 0, nr * sizeof(double), h->stream));
    SolveResult res;
    if ((rc = solve_pcg64(h, so, res))) return rc;
    if (res.status < 0) {
        h->err = "reference solve broke down";
        return res.status;
    }
    CK(cudaMemcpyAsync(h->x_star, h->sys.x, nr * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
    const int total = std::max(1, res.iterations);
    std::vector<int> snap;
    for (int k = 0; k < np; ++k) {
        const int it = np == 1 ? 0 : (int)std::floor(std::pow((double)total + 1.0, (double)k / (np - 1))) - 1;
        if (snap.empty() || it > snap.back()) snap.push_back(std::min(it, total - 1));
    }
    CK(cudaMemsetAsync(h->sys.x, 0, nr * sizeof(double), h->stream));
    CK(mh::launch_reset_ctl(h->sys, h->stream));
    CK(mh::launch_cg_init(h->sys, so.r_tol * so.r_tol, 0.0, total + 1, 0, h->stream));
    h->n_launch += 1;
    er.clear();
    int it = 0;
    for (int target : snap) {
        for (; it < target; ++it) {
            CK(mh::launch_cg_iteration(h->sys, 64, h->stream));
            h->n_launch += 2;
        }
        const int k = (int)er.size();
        float *pr = h->pair_r + (size_t)k * nr, *pe = h->pair_e + (size_t)k * nr;
        CK(mh::launch_pair_make(nr, h->x_star, h->sys.x, h->sys.r, pe, pr, h->pair_acc, h->stream));
        double acc[2];
        CK(cudaMemcpyAsync(acc, h->pair_acc, sizeof(acc), cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
        h->n_launch += 1;
        if (!(acc[0] > 0.0) || !(acc[1] > 0.0) || !std::isfinite(acc[0]) || !std::isfinite(acc[1])) continue;
        const double sc = 1.0 / std::sqrt(acc[0]);
        CK(mh::launch_pair_scale(nr, pe, pr, (float)sc, h->stream));
        h->n_launch += 1;
        er.push_back(acc[1] * sc * sc);
    }
    if (er.empty()) {
        h->err = "no usable training pair";
        return MH_ERR_STATE;
    }
    return MH_OK;
}

// Builds the training hierarchy of the current matrix (the network's inputs need the FP32
// scaled matrix and its features).
int training_setup(mh_handle *h) {
    int rc;
    if ((rc = ensure_learned(h)) || (rc = nn_weights(h))) return rc;
    if (h->sys.rows_per_thread != 1) {
        const int t[2] = {mh::krylov_target_blocks(1, 64), mh::krylov_target_blocks(1, 32)};
        if ((rc = apply_launch_shape(h, 1, t))) return rc;
    }
    h->amg.set_fine_weights(h->sn_w);
    cudaError_t e = h->amg.setup(h->sys, training_amg_options(h), h->stream);
    h->amg_epoch += 1;
    h->amg_matrix_epoch = -1;  // the next solve builds the solver's hierarchy again
    h->amg_training = true;
    h->tr_hier_epoch = h->matrix_epoch;
    if (e != cudaSuccess) {
        h->err = "AMG setup: " + h->amg.err;
        cudaGetLastError();
        return MH_ERR_CUDA;
    }
    return MH_OK;
}

int learned_train_impl(mh_handle *h, const mh_learn_opts &o, mh_learn_stats &st) {
    int rc;
    const int np = std::max(1, std::min(o.n_pairs, 64));
    if ((rc = ensure_learned(h)) || (rc = ensure_train(h, np))) return rc;
    const int64_t nr = h->sys.n_rows;
    cudaEvent_t e0 = h->ev[0], e1 = h->ev[1], e2 = h->ev[5];
    CK(cudaEventRecord(e0, h->stream));
    std::vector<double> er;
    if ((rc = make_pairs(h, np, o.solve_rtol, er))) return rc;
    const int n_ok = (int)er.size();
    CK(cudaEventRecord(e1, h->stream));
    if ((rc = training_setup(h))) return rc;
    // Adam, one step per pair, pairs shuffled every epoch
    const int epochs = std::max(1, o.epochs);
    const float lr = o.lr > 0.f ? o.lr : 2e-3f;
    std::mt19937_64 rng(o.seed);
    std::vector<int> order(n_ok);
    for (int k = 0; k < n_ok; ++k) order[k] = k;
    for (int ep = 0; ep < epochs; ++ep) {
        std::shuffle(order.begin(), order.end(), rng);
        double sum = 0.0;
        for (int k : order) {
            double l = 0.0;
            if ((rc = train_eval(h, h->pair_r + (size_t)k * nr, h->pair_e + (size_t)k * nr, er[k], true, &l))) {
                if (rc == MH_ERR_NONFINITE) h->err = "training loss is not finite";
                return rc;
            }
            sum += l;
            h->nn_step += 1;
            CK(mh::sn_adam(h->nn_w, h->nn_m, h->nn_v, h->nn_grad, h->nn_step, lr, h->stream));
            h->n_launch += 1;
        }
        if (ep == 0) st.loss_initial = sum / n_ok;
        if (ep == epochs - 1) st.loss_final = sum / n_ok;
    }
    h->sn_key_step = -1;  // the solver recomputes the weights with the trained network
    CK(cudaEventRecord(e2, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    st.ms_pairs = ms;
    CK(cudaEventElapsedTime(&ms, e1, e2));
    st.ms_train = ms;
    st.n_pairs = n_ok;
    st.epochs = epochs;
    return MH_OK;
}

int solve_impl(mh_handle *h, const mh_solve_opts *opts_in, mh_solve_stats *stats, bool have_guess_default) {
    mh_solve_opts o;
    mh_solve_opts_default(&o);
    if (opts_in) o = *opts_in;
    if (o.max_it <= 0) o.max_it = 20000;
    // the multigrid methods (plain or with the learned smoother) take long iterations and few
    // FP64 replacements
    const bool multigrid = o.method == MH_SOLVER_AMG || o.method == MH_SOLVER_FCG_LEARNED;
    if (o.iters_per_graph <= 0) o.iters_per_graph = multigrid ? 2 : 16;
    if (o.inner_max_it <= 0) o.inner_max_it = 2000;
    if (!(o.inner_rtol > 0.0)) o.inner_rtol = multigrid ? 1e-3 : 0.1;
    // MH_HOST_LOOP=1 makes the host-polled loop the default (profilers cannot see the kernels
    // inside a graph with conditional nodes)
    const char *hl = getenv("MH_HOST_LOOP");
    h->host_loop = o.host_loop != 0 || (hl && hl[0] == '1');
    if (!(o.r_tol >= 0.0)) o.r_tol = 1e-10;
    if (!(o.a_tol >= 0.0)) o.a_tol = 0.0;
    const bool guess = o.use_initial_guess || have_guess_default;
    const int64_t launches0 = h->n_launch;
    std::fill(h->inst_iters.begin(), h->inst_iters.end(), 0);
    std::fill(h->inst_status.begin(), h->inst_status.end(), 0);
    for (int k = 0; k < MH_KERNEL_CLASSES; ++k) {
        h->kernel_ms[k] = 0.0;
        h->kernel_count[k] = 0;
    }
    CK(cudaEventRecord(h->ev[2], h->stream));
    if (guess) {
        CK(mh::launch_scale_in(h->sys, h->sol + h->topo.n_sides() + h->mesh.n_el, h->stream));
        h->n_launch += 1;
    } else {
        CK(cudaMemsetAsync(h->sys.x, 0, h->sys.n_rows * sizeof(double), h->stream));
    }
    SolveResult res;
    int rc = MH_OK;
    switch (o.method) {
        case MH_SOLVER_PCG64: rc = solve_pcg64(h, o, res); break;
        case MH_SOLVER_IR32: rc = solve_ir32(h, o, res); break;
        case MH_SOLVER_CHEB: rc = solve_fcg(h, o, res, Pc::Cheb); break;
        case MH_SOLVER_FCG_LEARNED: rc = solve_fcg(h, o, res, Pc::Nn); break;
        case MH_SOLVER_AMG: rc = solve_fcg(h, o, res, Pc::Amg); break;
        default:
            h->err = "solver method not available";
            return MH_ERR_INVALID;
    }
    if (rc) return rc;
    if ((o.method == MH_SOLVER_AMG || o.method == MH_SOLVER_FCG_LEARNED) && h->amg.fine_tma_failed(h->stream)) {
        h->err = "multigrid: a fine-level shared-memory stage did not complete (bounded wait timed out)";
        return MH_ERR_CUDA;
    }
    if (res.status == MH_OK && res.fell_back) res.status = MH_FELL_BACK;
    CK(cudaEventRecord(h->ev[3], h->stream));
    CK(mh::launch_backsub(h->ed, h->as, h->sys, h->sol, h->topo.n_sides(), h->mesh.n_el, h->topo.n_edges(),
                          h->stream));
    CK(cudaEventRecord(h->ev[4], h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->n_launch += 1;
    for (int d = 1; d <= 3; ++d) h->n_launch += h->as.dim_count[d] > 0;
    h->solved = true;
    if (stats) {
        std::memset(stats, 0, sizeof(*stats));
        stats->status = res.status;
        stats->iterations = res.iterations;
        stats->outer_iterations = res.outer;
        stats->fell_back = res.fell_back;
        stats->rel_residual = res.rel;
        stats->rel_residual_unscaled = res.rel_orig;
        stats->kernel_launches = h->n_launch - launches0;
        for (int k = 0; k < MH_KERNEL_CLASSES; ++k) {
            stats->kernel_ms[k] = h->kernel_ms[k];
            stats->kernel_count[k] = h->kernel_count[k];
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, h->ev[2], h->ev[3]);
        stats->ms_solve = ms;
        cudaEventElapsedTime(&ms, h->ev[3], h->ev[4]);
        stats->ms_backsub = ms;
        stats->ms_assembly = h->ms_assembly;
        stats->ms_setup = res.ms_setup;
    }
    return res.status;
}

}  // namespace

extern "C" {

const char *mh_version(void) { return "mh-darcy-b200 0.1 (sm_100a)"; }

const char *mh_status_string(int s) {
    switch (s) {
        case MH_OK: return "ok";
        case MH_NOT_CONVERGED: return "not converged";
        case MH_FELL_BACK: return "converged after fallback";
        case MH_ERR_INVALID: return "invalid argument";
        case MH_ERR_SINGULAR: return "singular local matrix";
        case MH_ERR_CUDA: return "CUDA error";
        case MH_ERR_STATE: return "call out of order";
        case MH_ERR_NOMEM: return "out of memory";
        case MH_ERR_NONFINITE: return "non-finite value";
        case MH_ERR_TOPOLOGY: return "invalid mesh topology";
        case MH_ERR_BREAKDOWN: return "CG breakdown";
        case MH_ERR_IO: return "file cannot be read";
        default: return "unknown status";
    }
}

int mh_device_available(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n > 0 ? 1 : 0;
}

int mh_cube_mesh_create(int32_t n, int32_t n_planes, const int32_t *plane_axis, const int32_t *plane_index,
                        int32_t n_lines, const int32_t *line_axis, const int32_t *line_a, const int32_t *line_b,
                        mh_mesh **out) {
    if (!out || n_planes < 0 || n_lines < 0) return MH_ERR_INVALID;
    *out = nullptr;
    std::vector<int> pa, pi, la, l1, l2;
    for (int i = 0; i < n_planes; ++i) {
        pa.push_back(plane_axis[i]);
        pi.push_back(plane_index[i]);
    }
    for (int i = 0; i < n_lines; ++i) {
        la.push_back(line_axis[i]);
        l1.push_back(line_a[i]);
        l2.push_back(line_b[i]);
    }
    auto *m = new (std::nothrow) mh_mesh();
    if (!m) return MH_ERR_NOMEM;
    std::string err;
    int rc = mh::build_cube_mesh(n, pa, pi, la, l1, l2, m->m, &err);
    if (rc) {
        delete m;
        return rc;
    }
    *out = m;
    return MH_OK;
}

int mh_mesh_describe(const mh_mesh *m, mh_mesh_desc *d) {
    if (!m || !d) return MH_ERR_INVALID;
    d->n_nodes = m->m.n_nodes;
    d->node_xyz = m->m.xyz.data();
    d->n_elements = m->m.n_el;
    d->el_dim = m->m.dim.data();
    d->el_nodes = m->m.nodes.data();
    d->n_bc_elements = m->m.n_bc;
    d->bc_dim = m->m.bc_dim.data();
    d->bc_nodes = m->m.bc_nodes.data();
    return MH_OK;
}

void mh_mesh_destroy(mh_mesh *m) { delete m; }

void mh_solve_opts_default(mh_solve_opts *o) {
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->method = MH_SOLVER_PCG64;
    o->max_it = 20000;
    o->r_tol = 1e-10;
    o->a_tol = 0.0;
    o->use_initial_guess = 0;
    o->cheb_degree = 4;
    o->inner_rtol = 0.0;
    o->inner_max_it = 2000;
    o->iters_per_graph = 0;
}

}  // extern "C"

namespace {

bool desc_valid(const mh_mesh_desc *md) {
    if (!md || md->n_nodes <= 0 || md->n_elements <= 0 || !md->node_xyz || !md->el_dim || !md->el_nodes)
        return false;
    if (md->n_bc_elements < 0 || (md->n_bc_elements > 0 && (!md->bc_dim || !md->bc_nodes))) return false;
    return true;
}

// Appends a mesh to `m` (node indices shifted past the nodes already there).
void append_mesh(mh::MeshData &m, const mh_mesh_desc *md) {
    const int32_t shift = (int32_t)m.n_nodes;
    m.xyz.insert(m.xyz.end(), md->node_xyz, md->node_xyz + 3 * md->n_nodes);
    m.dim.insert(m.dim.end(), md->el_dim, md->el_dim + md->n_elements);
    for (int64_t k = 0; k < 4 * md->n_elements; ++k) {
        const int32_t v = md->el_nodes[k];
        m.nodes.push_back(v >= 0 ? v + shift : v);
    }
    if (md->n_bc_elements > 0) {
        m.bc_dim.insert(m.bc_dim.end(), md->bc_dim, md->bc_dim + md->n_bc_elements);
        for (int64_t k = 0; k < 4 * md->n_bc_elements; ++k) {
            const int32_t v = md->bc_nodes[k];
            m.bc_nodes.push_back(v >= 0 ? v + shift : v);
        }
    }
    m.n_nodes += md->n_nodes;
    m.n_el += md->n_elements;
    m.n_bc += md->n_bc_elements;
}

// Topology, edge-system layout and device set-up for a mesh whose instances own the element
// ranges inst_el (one instance: {0, n_el}).
int create_impl(mh_handle *h, const std::vector<int64_t> &inst, const mh_mortar_desc *mortar = nullptr) {
    mh::MeshData &m = h->mesh;
    if (!check_finite(m.xyz.data(), (int64_t)m.xyz.size())) return MH_ERR_NONFINITE;
    int rc = mh::build_topology(m, h->topo, &h->err);
    if (rc) return rc;
    const mh::Topology &t = h->topo;
    h->ngh_hi_el.resize(t.n_ngh());
    h->ngh_meas.resize(t.n_ngh());
    for (int64_t i = 0; i < t.n_ngh(); ++i) {
        int32_t side = t.ngh_side[i];
        int64_t e = std::upper_bound(t.el_side_start.begin(), t.el_side_start.end(), side) - t.el_side_start.begin() - 1;
        h->ngh_hi_el[i] = (int32_t)e;
        h->ngh_meas[i] = side_measure_host(m, e, side - t.el_side_start[e]);
    }
    int rpt = 1;  // best on B200 at cfg2 (R = 1/2/4 measured); mh_autotune can change it
    if (const char *env = getenv("MH_ROWS_PER_THREAD")) {
        int v = atoi(env);
        if (v == 1 || v == 2 || v == 4) rpt = v;
    }
    const int targets[2] = {mh::krylov_target_blocks(rpt, 64), mh::krylov_target_blocks(rpt, 32)};
    mh::ExtraBlocks extra;
    if (mortar && (rc = mh::mortar_blocks(m, h->topo, *mortar, extra, &h->err))) return rc;
    rc = mh::build_host_system(m, h->topo, inst, rpt, targets, h->hs, &h->err, extra.edges.empty() ? nullptr : &extra);
    if (rc) return rc;
    const int n_inst = (int)inst.size() - 1;
    h->inst_iters.assign(n_inst, 0);
    h->inst_status.assign(n_inst, 0);
    h->inst_rel.assign(n_inst, 0.0);
    return device_setup(h);
}

}  // namespace

extern "C" {

int mh_create(const mh_mesh_desc *md, mh_handle **out) {
    if (!out || !desc_valid(md)) return MH_ERR_INVALID;
    *out = nullptr;
    auto *h = new (std::nothrow) mh_handle();
    if (!h) return MH_ERR_NOMEM;
    append_mesh(h->mesh, md);
    int rc = create_impl(h, {0, h->mesh.n_el});
    if (rc) {
        mh_destroy(h);
        return rc;
    }
    *out = h;
    return MH_OK;
}

int mh_create_mortar(const mh_mesh_desc *md, const mh_mortar_desc *mortar, mh_handle **out) {
    if (!out || !desc_valid(md) || !mortar) return MH_ERR_INVALID;
    *out = nullptr;
    auto *h = new (std::nothrow) mh_handle();
    if (!h) return MH_ERR_NOMEM;
    append_mesh(h->mesh, md);
    int rc = create_impl(h, {0, h->mesh.n_el}, mortar);
    if (rc) {
        mh_destroy(h);
        return rc;
    }
    *out = h;
    return MH_OK;
}

int mh_create_batch(const mh_mesh_desc *meshes, int32_t n_inst, mh_handle **out) {
    if (!out || !meshes || n_inst <= 0) return MH_ERR_INVALID;
    *out = nullptr;
    for (int32_t i = 0; i < n_inst; ++i)
        if (!desc_valid(&meshes[i])) return MH_ERR_INVALID;
    auto *h = new (std::nothrow) mh_handle();
    if (!h) return MH_ERR_NOMEM;
    std::vector<int64_t> inst(1, 0);
    for (int32_t i = 0; i < n_inst; ++i) {
        append_mesh(h->mesh, &meshes[i]);
        inst.push_back(h->mesh.n_el);
    }
    int rc = create_impl(h, inst);
    if (rc) {
        mh_destroy(h);
        return rc;
    }
    *out = h;
    return MH_OK;
}

int mh_smoother_weights_set(mh_handle *h, const float *w, int64_t n) {
    int rc = need_device(h);
    if (rc) return rc;
    const int64_t ne = h->topo.n_edges();
    if (!w) {
        h->user_fine_w = false;
        return MH_OK;
    }
    if (n < ne) return MH_ERR_INVALID;
    for (int64_t g = 0; g < ne; ++g)
        if (!(w[g] > 0.f) || !std::isfinite(w[g])) {
            h->err = "smoother weights must be positive and finite";
            return MH_ERR_INVALID;
        }
    if (!h->d_fine_w && !(h->d_fine_w = dalloc<float>(h, h->sys.n_rows))) return MH_ERR_NOMEM;
    std::vector<float> rows(h->sys.n_rows, 1.f);
    for (int64_t g = 0; g < ne; ++g) rows[h->hs.edge_row[g]] = w[g];
    CK(cudaMemcpyAsync(h->d_fine_w, rows.data(), rows.size() * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->user_fine_w = true;
    if (h->amg.fine_smoother_weights() == h->d_fine_w) h->amg.set_fine_weights(nullptr);  // new values
    return MH_OK;
}

int mh_smoother_weights_get(const mh_handle *hc, float *w, int64_t n) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    const int64_t ne = h->topo.n_edges();
    if (!w || n < ne) return MH_ERR_INVALID;
    const float *cur = h->amg.fine_smoother_weights();
    if (!cur) {
        std::fill(w, w + ne, 1.f);
        return MH_OK;
    }
    std::vector<float> rows(h->sys.n_rows);
    CK(cudaMemcpyAsync(rows.data(), cur, rows.size() * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    for (int64_t g = 0; g < ne; ++g) w[g] = rows[h->hs.edge_row[g]];
    return MH_OK;
}

int mh_csr_create(int64_t n, const int32_t *row_ptr, const int32_t *col, mh_handle **out) {
    if (!out || n <= 0 || n > INT32_MAX || !row_ptr || !col) return MH_ERR_INVALID;
    *out = nullptr;
    auto *h = new (std::nothrow) mh_handle();
    if (!h) return MH_ERR_NOMEM;
    h->general = true;
    // no mesh: n edges, no sides, elements, boundary objects or neighbours
    h->topo.el_side_start.assign(1, 0);
    h->topo.el_ngh_start.assign(1, 0);
    h->topo.edge_side_start.assign(n + 1, 0);
    int rpt = 1;
    const int targets[2] = {mh::krylov_target_blocks(rpt, 64), mh::krylov_target_blocks(rpt, 32)};
    int rc = mh::build_host_system_csr(n, row_ptr, col, rpt, targets, h->hs, &h->err);
    if (!rc) {
        h->inst_iters.assign(1, 0);
        h->inst_status.assign(1, 0);
        h->inst_rel.assign(1, 0.0);
        rc = device_setup(h);
    }
    if (rc) {
        mh_destroy(h);
        return rc;
    }
    *out = h;
    return MH_OK;
}

int mh_csr_set_values(mh_handle *h, const double *val, const double *rhs) {
    if (!h || !h->general || !val || !rhs) return MH_ERR_INVALID;
    const mh::HostSystem &hs = h->hs;
    const int64_t n = h->topo.n_edges(), nnz = hs.nnz;
    if (!check_finite(val, nnz) || !check_finite(rhs, n)) {
        h->err = "non-finite matrix or right-hand side value";
        return MH_ERR_NONFINITE;
    }
    int64_t bad = n;  // the first row whose diagonal is not positive
#pragma omp parallel for schedule(static) reduction(min : bad) if (n > (1 << 16))
    for (int64_t r = 0; r < n; ++r)
        if (!(val[hs.csr_diag[r]] > 0.0)) bad = std::min(bad, r);
    if (bad < n) {
        h->err = "row " + std::to_string(bad) + " has a diagonal entry <= 0: not a positive definite system";
        return MH_ERR_INVALID;
    }
    int rc = need_device(h);
    if (rc) return rc;
    CK(cudaMemcpyAsync(h->d_csr_val, val, nnz * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(h->sys.b, rhs, n * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    k_scatter<<<(unsigned)((nnz + 255) / 256), 256, 0, h->stream>>>(nnz, h->d_csr_slot, h->d_csr_val, h->sys.val_raw);
    CK(cudaGetLastError());
    CK(mh::launch_scale(h->sys, 1, h->stream));
    h->n_launch += 4;
    CK(cudaStreamSynchronize(h->stream));
    h->assembled = true;
    h->rhs_stale = false;
    h->solved = false;
    h->matrix_epoch += 1;
    return MH_OK;
}

int mh_csr_get_solution(const mh_handle *hc, double *x, int64_t n) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    if (!h || !h->general || !x || n < h->topo.n_edges()) return MH_ERR_INVALID;
    int rc = need_device(h);
    if (rc) return rc;
    if (!h->solved) {
        h->err = "mh_solve must come before mh_csr_get_solution";
        return MH_ERR_STATE;
    }
    CK(cudaMemcpyAsync(x, h->sol, h->topo.n_edges() * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return MH_OK;
}

void mh_destroy(mh_handle *h) {
    if (!h) return;
    if (h->device) cudaDeviceSynchronize();
    for (auto &gp : h->graph)
        for (auto &g : gp)
            if (g) cudaGraphExecDestroy(g);
    for (auto &g : h->loop_graph)
        if (g) cudaGraphExecDestroy(g);
    for (auto &evs : h->prof_ev)
        for (auto e : evs) cudaEventDestroy(e);
    if (h->fcg_graph) cudaGraphExecDestroy(h->fcg_graph);
    for (auto &p : h->amg_prof) {
        for (auto e : p.cycle)
            if (e) cudaEventDestroy(e);
        for (auto e : p.smooth) cudaEventDestroy(e);
    }
    h->amg.release();
    for (void *p : h->allocs) cudaFree(p);
    for (auto &e : h->ev)
        if (e) cudaEventDestroy(e);
    if (h->h_done) cudaFreeHost(h->h_done);
    if (h->h_small) cudaFreeHost(h->h_small);
    if (h->own_stream) cudaStreamDestroy(h->own_stream);
    delete h;
}

int mh_get_sizes(const mh_handle *h, mh_sizes *o) {
    if (!h || !o) return MH_ERR_INVALID;
    std::memset(o, 0, sizeof(*o));
    o->n_nodes = h->mesh.n_nodes;
    o->n_elements = h->mesh.n_el;
    o->n_sides = h->topo.n_sides();
    o->n_edges = h->topo.n_edges();
    o->n_boundaries = h->topo.n_bdr();
    o->n_neighbours = h->topo.n_ngh();
    for (int d = 1; d <= 3; ++d) o->n_el_dim[d] = (int64_t)h->hs.dim_list[d].size();
    o->mh_size = o->n_sides + o->n_elements + o->n_edges;
    o->schur_nnz = h->hs.nnz;
    o->sell_slots = h->hs.n_slots;
    o->n_rows_padded = h->hs.n_rows;
    o->n_instances = (int64_t)h->hs.inst_el.size() - 1;
    return MH_OK;
}

int mh_get_topology(const mh_handle *h, int32_t *el_side_start, int32_t *side_edge, int32_t *side_bdr,
                    int32_t *bdr_bc_element, int32_t *bdr_edge, int32_t *ngh_element, int32_t *ngh_edge,
                    int32_t *ngh_side) {
    if (!h) return MH_ERR_INVALID;
    const mh::Topology &t = h->topo;
    auto cp = [](int32_t *dst, const std::vector<int32_t> &v) {
        if (dst && !v.empty()) std::memcpy(dst, v.data(), v.size() * sizeof(int32_t));
    };
    cp(el_side_start, t.el_side_start);
    cp(side_edge, t.side_edge);
    cp(side_bdr, t.side_bdr);
    cp(bdr_bc_element, t.bdr_bc_el);
    cp(bdr_edge, t.bdr_edge);
    cp(ngh_element, t.ngh_el);
    cp(ngh_edge, t.ngh_edge);
    cp(ngh_side, t.ngh_side);
    return MH_OK;
}

int mh_set_coeffs(mh_handle *h, const mh_coeffs *c) {
    int rc = need_device(h);
    if (rc) return rc;
    if (h->general) {
        h->err = "the handle holds a general system (mh_csr_create): it has no mesh data";
        return MH_ERR_STATE;
    }
    if (!c) return MH_ERR_INVALID;
    const int64_t n = h->mesh.n_el;
    const double *arrs[6] = {c->conductivity, c->cross_section, c->sigma, c->water_source_density, c->storativity,
                             nullptr};
    for (int i = 0; i < 5; ++i)
        if (!check_finite(arrs[i], n)) return MH_ERR_NONFINITE;
    if (c->anisotropy && !check_finite(c->anisotropy, 9 * n)) return MH_ERR_NONFINITE;
    if (!check_positive(c->conductivity, n)) {
        h->err = "conductivity must be positive";
        return MH_ERR_INVALID;
    }
    if (!check_positive(c->cross_section, n)) {
        h->err = "cross_section must be positive";
        return MH_ERR_INVALID;
    }
    mh::ElemData &d = h->ed;
    if ((rc = fill_or_default(h, (double *)d.conductivity, c->conductivity, n, 1.0)) ||
        (rc = fill_or_default(h, (double *)d.cross_section, c->cross_section, n, 1.0)) ||
        (rc = fill_or_default(h, (double *)d.sigma, c->sigma, n, 1.0)) ||
        (rc = fill_or_default(h, (double *)d.source, c->water_source_density, n, 0.0)) ||
        (rc = fill_or_default(h, (double *)d.storativity, c->storativity, n, 1.0)))
        return rc;
    if (c->anisotropy) {
        if (!h->d_aniso) {
            h->d_aniso = dalloc<double>(h, 9 * n);
            if (!h->d_aniso) return MH_ERR_NOMEM;
        }
        CK(cudaMemcpyAsync(h->d_aniso, c->anisotropy, 9 * n * sizeof(double), cudaMemcpyHostToDevice, h->stream));
        d.anisotropy = h->d_aniso;
    } else {
        d.anisotropy = nullptr;
    }
    CK(cudaStreamSynchronize(h->stream));
    h->coeffs_set = true;
    h->assembled = false;
    h->solved = false;  // the post-processing needs a solution of the new coefficients
    return MH_OK;
}

int mh_set_bc(mh_handle *h, const mh_bc *bc) {
    int rc = need_device(h);
    if (rc) return rc;
    if (h->general) {
        h->err = "the handle holds a general system (mh_csr_create): it has no mesh data";
        return MH_ERR_STATE;
    }
    if (!bc) return MH_ERR_INVALID;
    const int64_t n = h->topo.n_bdr();
    if (bc->type)
        for (int64_t i = 0; i < n; ++i)
            if (bc->type[i] < MH_BC_NONE || bc->type[i] > MH_BC_ROBIN) {
                h->err = "unknown boundary condition type";
                return MH_ERR_INVALID;
            }
    if (!check_finite(bc->pressure, n) || !check_finite(bc->flux, n) || !check_finite(bc->robin_sigma, n))
        return MH_ERR_NONFINITE;
    mh::ElemData &d = h->ed;
    if (bc->type) {
        CK(cudaMemcpyAsync((void *)d.bc_type, bc->type, n * sizeof(int32_t), cudaMemcpyHostToDevice, h->stream));
    } else {
        CK(cudaMemsetAsync((void *)d.bc_type, 0, n * sizeof(int32_t), h->stream));
    }
    if ((rc = fill_or_default(h, (double *)d.bc_pressure, bc->pressure, n, 0.0)) ||
        (rc = fill_or_default(h, (double *)d.bc_flux, bc->flux, n, 0.0)) ||
        (rc = fill_or_default(h, (double *)d.bc_sigma, bc->robin_sigma, n, 0.0)))
        return rc;
    CK(cudaStreamSynchronize(h->stream));
    // boundary types and Robin coefficients enter the matrix, pressures and fluxes only the
    // right-hand side: an unsteady step after a change of values alone reassembles the rhs
    std::vector<int32_t> typ(n, 0);
    std::vector<double> sig(n, 0.0);
    if (bc->type) std::copy(bc->type, bc->type + n, typ.begin());
    if (bc->robin_sigma) std::copy(bc->robin_sigma, bc->robin_sigma + n, sig.begin());
    const bool matrix_same = h->bc_set && typ == h->bc_type_host && sig == h->bc_sigma_host;
    h->bc_type_host.swap(typ);
    h->bc_sigma_host.swap(sig);
    h->bc_set = true;
    if (!matrix_same) h->assembled = false;
    h->rhs_stale = true;
    return MH_OK;
}

int mh_assemble(mh_handle *h) {
    int rc = need_device(h);
    if (rc) return rc;
    if (h->general) {
        h->err = "the handle holds a general system (mh_csr_create): it has no mesh data";
        return MH_ERR_STATE;
    }
    if (!h->coeffs_set || !h->bc_set) {
        h->err = "mh_set_coeffs and mh_set_bc must come before mh_assemble";
        return MH_ERR_STATE;
    }
    return assemble_impl(h, 3);
}

int mh_solve(mh_handle *h, const mh_solve_opts *opts, mh_solve_stats *stats) {
    int rc = need_device(h);
    if (rc) return rc;
    if (!h->assembled || h->rhs_stale) {
        h->err = "mh_assemble must come before mh_solve";
        return MH_ERR_STATE;
    }
    return solve_impl(h, opts, stats, false);
}

int mh_get_solution(const mh_handle *hc, double *out, int64_t len) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    const int64_t msize = h->topo.n_sides() + h->mesh.n_el + h->topo.n_edges();
    if (!out || len < msize) return MH_ERR_INVALID;
    CK(cudaMemcpyAsync(out, h->sol, msize * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return MH_OK;
}

int mh_get_solution_device(const mh_handle *hc, double *dev_out, int64_t len) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    const int64_t msize = h->topo.n_sides() + h->mesh.n_el + h->topo.n_edges();
    if (!dev_out || len < msize) return MH_ERR_INVALID;
    CK(cudaMemcpyAsync(dev_out, h->sol, msize * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return MH_OK;
}

// make_element_vector (darcy_flow_mh_output.cc:301-323) on the device, into dev_out [3 n_el]
static int element_flux_into(mh_handle *h, double *dev_out) {
    if (!h->solved) {
        h->err = "no solution of the current coefficients: mh_solve or mh_unsteady_step must come before the element fluxes";
        return MH_ERR_STATE;
    }
    CK(mh::launch_element_flux(h->ed, h->as, h->sol, dev_out, h->stream));
    return MH_OK;
}

int mh_get_element_flux(const mh_handle *hc, double *out, int64_t len) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    const int64_t n = 3 * h->mesh.n_el;
    if (!out || len < n) return MH_ERR_INVALID;
    if (!h->d_elflux) {
        h->d_elflux = dalloc<double>(h, std::max<int64_t>(n, 1));
        if (!h->d_elflux) return MH_ERR_NOMEM;
    }
    if ((rc = element_flux_into(h, h->d_elflux))) return rc;
    CK(cudaMemcpyAsync(out, h->d_elflux, n * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return MH_OK;
}

int mh_get_element_flux_device(const mh_handle *hc, double *dev_out, int64_t len) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    if (!dev_out || len < 3 * h->mesh.n_el) return MH_ERR_INVALID;
    if ((rc = element_flux_into(h, dev_out))) return rc;
    CK(cudaStreamSynchronize(h->stream));
    return MH_OK;
}

int mh_get_node_pressure(const mh_handle *hc, double *out, int64_t len) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    const int64_t nn = h->mesh.n_nodes, ne = h->mesh.n_el;
    if (!out || len < nn) return MH_ERR_INVALID;
    if (!h->solved) {
        h->err = "no solution of the current coefficients: mh_solve or mh_unsteady_step must come before the node pressures";
        return MH_ERR_STATE;
    }
    if (!h->d_node_p) {
        // node -> element incidence (elements ascending), once per mesh
        std::vector<int32_t> start(nn + 1, 0), inc;
        for (int64_t e = 0; e < ne; ++e)
            for (int32_t k = 0; k <= h->mesh.dim[e]; ++k) start[h->mesh.nodes[4 * e + k] + 1]++;
        for (int64_t v = 0; v < nn; ++v) start[v + 1] += start[v];
        inc.resize(start[nn]);
        std::vector<int32_t> fill(start.begin(), start.end() - 1);
        for (int64_t e = 0; e < ne; ++e)
            for (int32_t k = 0; k <= h->mesh.dim[e]; ++k) inc[fill[h->mesh.nodes[4 * e + k]]++] = (int32_t)e;
        if ((rc = upload(h, h->d_node_inc_start, start)) || (rc = upload(h, h->d_node_inc, inc))) return rc;
        h->d_node_p = dalloc<double>(h, std::max<int64_t>(nn, 1));
        if (!h->d_node_p) return MH_ERR_NOMEM;
    }
    CK(mh::launch_node_pressure(h->ed, h->d_node_inc_start, h->d_node_inc, nn, h->sol, h->topo.n_sides(), ne,
                                h->d_node_p, h->stream));
    CK(cudaMemcpyAsync(out, h->d_node_p, nn * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return MH_OK;
}

// Items of one kind grouped by region (ascending within a region), cut into chunks of at most
// kBalanceChunkItems: items, chunk begins [n_chunks+1] and region-chunk offsets [n_reg+1].
static void group_by_region(const std::vector<int32_t> &item_region, const std::vector<int32_t> &item_id,
                            int32_t n_reg, std::vector<int32_t> &items, std::vector<int64_t> &chunk_begin,
                            std::vector<int64_t> &region_chunk) {
    std::vector<int64_t> off(n_reg + 1, 0);
    for (int32_t r : item_region) off[r + 1]++;
    for (int32_t r = 0; r < n_reg; ++r) off[r + 1] += off[r];
    items.assign(item_id.size(), 0);
    std::vector<int64_t> fill(off.begin(), off.end() - 1);
    for (size_t i = 0; i < item_id.size(); ++i) items[fill[item_region[i]]++] = item_id[i];
    chunk_begin.assign(1, 0);
    region_chunk.assign(1, 0);
    for (int32_t r = 0; r < n_reg; ++r) {
        for (int64_t b = off[r]; b < off[r + 1]; b += mh::kBalanceChunkItems)
            chunk_begin.push_back(std::min(off[r + 1], b + mh::kBalanceChunkItems));
        region_chunk.push_back((int64_t)chunk_begin.size() - 1);
    }
}

int mh_water_balance(const mh_handle *hc, const int32_t *bdr_region, int32_t n_bdr_regions,
                     const int32_t *el_region, int32_t n_el_regions, double *bdr_out, double *src_out) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    const int64_t nb = h->topo.n_bdr(), ne = h->mesh.n_el, ns = h->topo.n_sides();
    if (!bdr_region || !el_region || !bdr_out || !src_out || n_bdr_regions < 1 || n_el_regions < 1)
        return MH_ERR_INVALID;
    for (int64_t b = 0; b < nb; ++b)
        if (bdr_region[b] < 0 || bdr_region[b] >= n_bdr_regions) {
            h->err = "boundary region index out of range";
            return MH_ERR_INVALID;
        }
    for (int64_t e = 0; e < ne; ++e)
        if (el_region[e] < 0 || el_region[e] >= n_el_regions) {
            h->err = "element region index out of range";
            return MH_ERR_INVALID;
        }
    if (!h->solved) {
        h->err = "no solution of the current coefficients: mh_solve or mh_unsteady_step must come before the water balance";
        return MH_ERR_STATE;
    }
    // boundary sides (ascending) and elements, grouped by region
    std::vector<int32_t> reg, ids, bitems, sitems;
    std::vector<int64_t> bchunk, breg, schunk, sreg;
    for (int64_t sd = 0; sd < ns; ++sd) {
        const int32_t b = h->topo.side_bdr[sd];
        if (b < 0) continue;
        reg.push_back(bdr_region[b]);
        ids.push_back((int32_t)sd);
    }
    group_by_region(reg, ids, n_bdr_regions, bitems, bchunk, breg);
    reg.assign(el_region, el_region + ne);
    ids.resize(ne);
    for (int64_t e = 0; e < ne; ++e) ids[e] = (int32_t)e;
    group_by_region(reg, ids, n_el_regions, sitems, schunk, sreg);
    const int64_t n_items = (int64_t)bitems.size() + (int64_t)sitems.size();
    const int64_t n_index = (int64_t)(bchunk.size() + breg.size() + schunk.size() + sreg.size());
    const int64_t nbc = (int64_t)bchunk.size() - 1, nsc = (int64_t)schunk.size() - 1;
    const int64_t need = 3 * nbc + nsc + 3 * (int64_t)n_bdr_regions + n_el_regions;
    if (n_items > h->bal_items_cap) {
        if (!(h->d_bal_items = dalloc<int32_t>(h, n_items))) return MH_ERR_NOMEM;
        h->bal_items_cap = n_items;
    }
    if (n_index > h->bal_index_cap) {
        if (!(h->d_bal_index = dalloc<int64_t>(h, n_index))) return MH_ERR_NOMEM;
        h->bal_index_cap = n_index;
    }
    if (need > h->balance_cap) {
        if (!(h->d_balance = dalloc<double>(h, need))) return MH_ERR_NOMEM;
        h->balance_cap = need;
    }
    std::vector<int32_t> hitems(bitems);
    hitems.insert(hitems.end(), sitems.begin(), sitems.end());
    std::vector<int64_t> hindex(bchunk);
    hindex.insert(hindex.end(), breg.begin(), breg.end());
    hindex.insert(hindex.end(), schunk.begin(), schunk.end());
    hindex.insert(hindex.end(), sreg.begin(), sreg.end());
    if (n_items > 0)
        CK(cudaMemcpyAsync(h->d_bal_items, hitems.data(), n_items * sizeof(int32_t), cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(h->d_bal_index, hindex.data(), n_index * sizeof(int64_t), cudaMemcpyHostToDevice, h->stream));
    mh::BalanceLists L;
    L.bdr_items = h->d_bal_items;
    L.src_items = h->d_bal_items + bitems.size();
    L.bdr_chunk_begin = h->d_bal_index;
    L.bdr_region_chunk = L.bdr_chunk_begin + bchunk.size();
    L.src_chunk_begin = L.bdr_region_chunk + breg.size();
    L.src_region_chunk = L.src_chunk_begin + schunk.size();
    L.n_bdr_chunks = nbc;
    L.n_src_chunks = nsc;
    L.n_bdr_reg = n_bdr_regions;
    L.n_src_reg = n_el_regions;
    double *bo = h->d_balance + 3 * nbc + nsc, *so = bo + 3 * (int64_t)n_bdr_regions;
    CK(mh::launch_water_balance(h->ed, h->sol, L, h->d_balance, bo, so, h->stream));
    CK(cudaMemcpyAsync(bdr_out, bo, 3 * (size_t)n_bdr_regions * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(src_out, so, (size_t)n_el_regions * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return MH_OK;
}

// The convection matrix's sparsity pattern (ConvectionTransport::create_transport_matrix_mpi,
// transport.cc:788-923, with the entries written in its order): per element row the diagonal,
// for each side that is not on a boundary object every other side of its edge, for each VB
// neighbour (the row element lower-dimensional) the higher element, and for each VB coupling in
// which the row element is the higher one the lower element.  Slots are sorted by column; two
// slots of one row never share a column in a simplicial mesh (two elements share at most one
// face, a VB pair one side), which is checked.
static int build_transport_pattern(mh_handle *h) {
    const mh::Topology &t = h->topo;
    const int64_t ne = h->mesh.n_el, ns = t.n_sides();
    std::vector<int32_t> side_el(ns);
    for (int64_t e = 0; e < ne; ++e)
        for (int32_t k = t.el_side_start[e]; k < t.el_side_start[e + 1]; ++k) side_el[k] = (int32_t)e;
    struct Slot {
        int32_t col, kind, a, b;
    };
    std::vector<std::vector<Slot>> rows(ne);
    for (int64_t i = 0; i < ne; ++i) {
        auto &r = rows[i];
        r.push_back({(int32_t)i, mh::kTrDiag, -1, -1});
        for (int32_t si = t.el_side_start[i]; si < t.el_side_start[i + 1]; ++si) {
            if (t.side_bdr[si] >= 0) continue;
            const int32_t ed = t.side_edge[si];
            for (int32_t k = t.edge_side_start[ed]; k < t.edge_side_start[ed + 1]; ++k) {
                const int32_t so = t.edge_sides[k];
                if (so != si) r.push_back({side_el[so], mh::kTrEdge, si, so});
            }
        }
        for (int32_t k = t.el_ngh_start[i]; k < t.el_ngh_start[i + 1]; ++k) {
            const int32_t hs = t.ngh_side[t.el_ngh[k]];
            r.push_back({side_el[hs], mh::kTrVbLower, hs, -1});
            rows[side_el[hs]].push_back({(int32_t)i, mh::kTrVbHigher, hs, -1});
        }
    }
    std::vector<int32_t> rp(ne + 1, 0), col, kind, sa, sb;
    for (int64_t i = 0; i < ne; ++i) {
        auto &r = rows[i];
        std::sort(r.begin(), r.end(), [](const Slot &x, const Slot &y) { return x.col < y.col; });
        for (size_t k = 0; k < r.size(); ++k) {
            if (k && r[k].col == r[k - 1].col) {
                h->err = "convection matrix: two couplings of one element pair (degenerate mesh)";
                return MH_ERR_TOPOLOGY;
            }
            col.push_back(r[k].col);
            kind.push_back(r[k].kind);
            sa.push_back(r[k].a);
            sb.push_back(r[k].b);
        }
        rp[i + 1] = (int32_t)col.size();
    }
    mh::TransportPattern &p = h->conv;
    p.n_el = ne;
    p.n_edges = t.n_edges();
    p.nnz = (int64_t)col.size();
    int rc;
    if ((rc = upload(h, p.row_ptr, rp)) || (rc = upload(h, p.kind, kind)) || (rc = upload(h, p.slot_a, sa)) ||
        (rc = upload(h, p.slot_b, sb)) || (rc = upload(h, p.edge_start, t.edge_side_start)) ||
        (rc = upload(h, p.edge_sides, t.edge_sides)) || (rc = upload(h, p.ngh_side, t.ngh_side)))
        return rc;
    p.edge_flow = dalloc<double>(h, std::max<int64_t>(p.n_edges, 1));
    p.diag_max = dalloc<unsigned long long>(h, 1);
    h->d_tr_val = dalloc<double>(h, std::max<int64_t>(p.nnz, 1));
    h->d_tr_por = dalloc<double>(h, std::max<int64_t>(ne, 1));
    if (!p.edge_flow || !p.diag_max || !h->d_tr_val || !h->d_tr_por) return MH_ERR_NOMEM;
    h->tr_row_ptr.swap(rp);
    h->tr_col.swap(col);
    h->tr_built = true;
    return MH_OK;
}

// values of the convection matrix into dev_val for the last solution; cfl = 1 / max |a_ii|
static int transport_values(mh_handle *h, const double *dev_porosity, double *dev_val, double *cfl) {
    if (!h->solved) {
        h->err = "no solution of the current coefficients: mh_solve or mh_unsteady_step must come before the convection matrix";
        return MH_ERR_STATE;
    }
    CK(mh::launch_transport_matrix(h->ed, h->conv, dev_porosity, h->sol, dev_val, h->stream));
    unsigned long long bits = 0;
    if (int rc = read_back(h, &bits, h->conv.diag_max, sizeof(bits))) return rc;
    if (cfl) {
        double mx;
        std::memcpy(&mx, &bits, sizeof(mx));
        *cfl = mx > 0.0 ? 1.0 / mx : std::numeric_limits<double>::infinity();
    }
    return MH_OK;
}

int mh_transport_matrix(const mh_handle *hc, const double *porosity, int64_t *nnz, int32_t *row_ptr, int32_t *col,
                        double *val, double *cfl_max_step) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    if (!nnz) return MH_ERR_INVALID;
    if (!h->tr_built && (rc = build_transport_pattern(h))) return rc;
    *nnz = h->conv.nnz;
    if (!row_ptr && !col && !val && !cfl_max_step) return MH_OK;  // the size query
    const int64_t ne = h->mesh.n_el;
    if (porosity && !check_finite(porosity, ne)) return MH_ERR_NONFINITE;
    if (porosity && !check_positive(porosity, ne)) {
        h->err = "porosity must be positive";
        return MH_ERR_INVALID;
    }
    if (porosity) CK(cudaMemcpyAsync(h->d_tr_por, porosity, ne * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    if ((rc = transport_values(h, porosity ? h->d_tr_por : nullptr, h->d_tr_val, cfl_max_step))) return rc;
    if (row_ptr) std::memcpy(row_ptr, h->tr_row_ptr.data(), (ne + 1) * sizeof(int32_t));
    if (col) std::memcpy(col, h->tr_col.data(), h->conv.nnz * sizeof(int32_t));
    if (val) {
        CK(cudaMemcpyAsync(val, h->d_tr_val, h->conv.nnz * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
        CK(cudaStreamSynchronize(h->stream));
    }
    return MH_OK;
}

int mh_transport_matrix_device(const mh_handle *hc, const double *dev_porosity, double *dev_val, int64_t len,
                               double *cfl_max_step) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    if (!h->tr_built && (rc = build_transport_pattern(h))) return rc;
    if (!dev_val || len < h->conv.nnz) return MH_ERR_INVALID;
    return transport_values(h, dev_porosity, dev_val, cfl_max_step);
}

int mh_get_schur_system(const mh_handle *hc, int32_t *row_ptr, int32_t *col, double *val, double *rhs) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    if (!h->assembled || h->rhs_stale) return MH_ERR_STATE;
    const HostSystem &hs = h->hs;
    std::vector<double> v(hs.n_slots), b(hs.n_rows);
    CK(cudaMemcpyAsync(v.data(), h->sys.val_raw, hs.n_slots * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(b.data(), h->sys.b, hs.n_rows * sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    const int64_t ne = h->topo.n_edges();
    int64_t k = 0;
    if (row_ptr) row_ptr[0] = 0;
    for (int64_t e = 0; e < ne; ++e) {
        const int64_t r = hs.edge_row[e];
        const int64_t sl = r / mh::kSliceRowsHost, lane = r % mh::kSliceRowsHost;
        const int64_t off = hs.slice_off[sl];
        for (int64_t j = 0; j < hs.row_ptr[r + 1] - hs.row_ptr[r]; ++j) {
            const int32_t c = hs.row_col[hs.row_ptr[r] + j];
            if (col) col[k] = hs.row_edge[c];
            if (val) val[k] = v[off + mh::sell_pos(r, c, j) * mh::kSliceRowsHost + lane];
            ++k;
        }
        if (row_ptr) row_ptr[e + 1] = (int32_t)k;
        if (rhs) rhs[e] = b[r];
    }
    return MH_OK;
}

int mh_unsteady_init(mh_handle *h, int32_t lumped, double dt, const double *init_pressure) {
    int rc = need_device(h);
    if (rc) return rc;
    if (!(dt > 0.0) || !std::isfinite(dt)) return MH_ERR_INVALID;
    if (!h->coeffs_set || !h->bc_set) return MH_ERR_STATE;
    const int64_t n_el = h->mesh.n_el, ns = h->topo.n_sides(), ne = h->topo.n_edges();
    if (init_pressure && !check_finite(init_pressure, n_el)) return MH_ERR_NONFINITE;
    // the previous step's solution: zero but for the initial element pressures (MH) or the edge
    // pressures they give (LMH)
    const size_t bytes = (size_t)(ns + n_el + ne) * sizeof(double);
    CK(cudaMemsetAsync(h->sol_prev, 0, bytes, h->stream));
    std::vector<double> edge;
    if (init_pressure && !lumped) {
        CK(cudaMemcpyAsync(h->sol_prev + ns, init_pressure, n_el * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    } else if (init_pressure) {
        // DarcyFlowLMH_Unsteady::setup_time_term: edge value += init / n_sides per side
        edge.assign(ne, 0.0);
        for (int64_t e = 0; e < n_el; ++e) {
            const int n = h->mesh.dim[e] + 1;
            for (int i = 0; i < n; ++i) edge[h->topo.side_edge[h->topo.el_side_start[e] + i]] += init_pressure[e] / n;
        }
        CK(cudaMemcpyAsync(h->sol_prev + ns + n_el, edge.data(), ne * sizeof(double), cudaMemcpyHostToDevice, h->stream));
    }
    CK(cudaMemcpyAsync(h->sol, h->sol_prev, bytes, cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    h->time_mode = lumped ? 2 : 1;
    h->ed.time_mode = h->time_mode;
    h->dt = dt;
    h->ed.dt = dt;
    return assemble_impl(h, 3);
}

int mh_unsteady_step(mh_handle *h, double dt, const mh_solve_opts *opts, mh_solve_stats *stats) {
    int rc = need_device(h);
    if (rc) return rc;
    if (h->time_mode == 0) return MH_ERR_STATE;
    if (!(dt > 0.0) || !std::isfinite(dt)) return MH_ERR_INVALID;
    if (dt != h->dt || !h->assembled) {
        h->dt = dt;
        h->ed.dt = dt;
        rc = assemble_impl(h, 3);
    } else {
        rc = assemble_impl(h, 2);  // matrix unchanged: only the time-term rhs moves
    }
    if (rc) return rc;
    int st = solve_impl(h, opts, stats, true);
    if (st < 0) return st;
    const int64_t msize = h->topo.n_sides() + h->mesh.n_el + h->topo.n_edges();
    CK(cudaMemcpyAsync(h->sol_prev, h->sol, msize * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return st;
}

const char *mh_last_error(const mh_handle *h) { return h ? h->err.c_str() : "null handle"; }

int mh_get_instance_offsets(const mh_handle *h, int64_t *el_off, int64_t *side_off, int64_t *edge_off,
                            int64_t *bdr_off) {
    if (!h) return MH_ERR_INVALID;
    const mh::HostSystem &hs = h->hs;
    const mh::Topology &t = h->topo;
    const int n = (int)hs.inst_el.size() - 1;
    for (int i = 0; i <= n; ++i) {
        if (el_off) el_off[i] = hs.inst_el[i];
        if (side_off) side_off[i] = t.el_side_start[hs.inst_el[i]];
        if (edge_off) edge_off[i] = hs.inst_edge[i];
    }
    if (bdr_off) {
        // boundary objects follow the instances' elements (edge ranges are per instance)
        int64_t b = 0;
        for (int i = 0; i < n; ++i) {
            bdr_off[i] = b;
            while (b < t.n_bdr() && t.bdr_edge[b] < hs.inst_edge[i + 1]) ++b;
        }
        bdr_off[n] = t.n_bdr();
    }
    return MH_OK;
}

int mh_get_instance_stats(const mh_handle *h, int32_t *iterations, double *rel_residual, int32_t *status) {
    if (!h) return MH_ERR_INVALID;
    const size_t n = h->inst_iters.size();
    for (size_t i = 0; i < n; ++i) {
        if (iterations) iterations[i] = h->inst_iters[i];
        if (rel_residual) rel_residual[i] = h->inst_rel[i];
        if (status) status[i] = h->inst_status[i];
    }
    return MH_OK;
}

int mh_autotune_ex(mh_handle *h, int32_t iterations, mh_tune_result *out) {
    if (!out) return MH_ERR_INVALID;
    std::memset(out, 0, sizeof(*out));
    int32_t R = 0;
    double us[2] = {0.0, 0.0};
    int rc = mh_autotune(h, iterations, &R, us);
    if (rc) return rc;
    out->rows_per_thread = R;
    out->us_per_iter_fp32 = us[0];
    out->us_per_iter_fp64 = us[1];
    // K1's element group: each candidate assembles the matrix and rhs three times (the same
    // values again), the fastest median wins
    double best = 1e300;
    int best_g = h->k1_group;
    for (int G : {64, 128, 256}) {
        if (h->general) break;  // a general CSR system has no element assembly
        float t[3];
        for (float &tk : t) {
            CK(cudaEventRecord(h->ev[0], h->stream));
            CK(mh::launch_local_blocks(h->ed, h->as, 3, G, h->stream));
            CK(mh::launch_gather(h->as, h->sys, 3, h->stream));
            CK(cudaEventRecord(h->ev[1], h->stream));
            CK(cudaEventSynchronize(h->ev[1]));
            CK(cudaEventElapsedTime(&tk, h->ev[0], h->ev[1]));
            for (int d = 1; d <= 3; ++d) h->n_launch += h->as.dim_count[d] > 0;
            h->n_launch += 1 + (h->as.n_add > 0);
        }
        std::sort(t, t + 3);
        if (1e3 * t[1] < best) {
            best = 1e3 * t[1];
            best_g = G;
        }
    }
    h->k1_group = best_g;
    out->k1_group = h->general ? 0 : best_g;
    out->us_assembly = h->general ? 0.0 : best;
    out->sell_rows_per_warp = 32 * R;
    // the multigrid's pairing passes from the fine level (aggregates of up to 4 or 8 fine rows):
    // which one converges faster depends on the system (hub-dominated fractured systems gain
    // from the larger aggregates, smooth ones lose), so each is timed on this system: two
    // complete solves to 1e-10 with the hierarchy rebuilt for each, the faster of the two kept
    // unless MH_AMG_PASSES fixes the count
    if (!getenv("MH_AMG_PASSES")) {
        double best_ms = 1e300;
        int best_p = 2;
        for (int p : {2, 3}) {
            h->amg_fine_passes = p;
            double t_min = 1e300;
            for (int rep = 0; rep < 2; ++rep) {
                mh_solve_opts so;
                mh_solve_opts_default(&so);
                so.method = MH_SOLVER_AMG;
                so.r_tol = 1e-10;
                mh_solve_stats st;
                std::memset(&st, 0, sizeof(st));
                h->amg_matrix_epoch = -1;  // the setup is part of what is timed
                const auto t0 = std::chrono::steady_clock::now();
                rc = solve_impl(h, &so, &st, false);
                const double ms =
                    std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
                if (rc < 0) return rc;
                if (st.status == MH_OK || st.status == MH_FELL_BACK) t_min = std::min(t_min, ms);
            }
            if (t_min < best_ms) {
                best_ms = t_min;
                best_p = p;
            }
        }
        h->amg_fine_passes = best_p;
        h->amg_matrix_epoch = -1;  // the next solve builds the hierarchy with the choice
        out->amg_fine_passes = best_p;
        out->ms_amg_solve = best_ms < 1e299 ? best_ms : 0.0;
    }
    return MH_OK;
}

int mh_autotune(mh_handle *h, int32_t iterations, int32_t *rows_per_thread, double *us_per_iter) {
    int rc = need_device(h);
    if (rc) return rc;
    if (!h->assembled) return MH_ERR_STATE;
    if (iterations <= 0) iterations = 64;
    const int ipg = 16;
    iterations = ((iterations + ipg - 1) / ipg) * ipg;
    double best = 1e300, best32 = 0.0, best64 = 0.0;
    int best_r = h->hs.rows_per_thread;
    std::vector<double> sums;
    for (int R : {1, 2, 4}) {
        const int targets[2] = {mh::krylov_target_blocks(R, 64), mh::krylov_target_blocks(R, 32)};
        if ((rc = apply_launch_shape(h, R, targets))) return rc;
        double t[2] = {0.0, 0.0};
        for (int k = 0; k < 2; ++k) {
            const int prec = k == 0 ? 64 : 32;
            // a fixed number of iterations from the current rhs (tolerance 0: never converges)
            CK(cudaMemsetAsync(h->sys.x, 0, h->sys.n_rows * sizeof(double), h->stream));
            CK(mh::launch_reset_ctl(h->sys, h->stream));
            if (prec == 64) {
                CK(mh::launch_cg_init(h->sys, 0.0, 0.0, iterations, 0, h->stream));
            } else {
                if ((rc = true_residual(h, sums))) return rc;
                for (int i = 0; i < h->sys.n_inst; ++i) sums[mh::kSumStride * i + mh::kSumActive] = 1.0;
                CK(cudaMemcpyAsync(h->sys.inst_sums, sums.data(), sizeof(double) * sums.size(),
                                   cudaMemcpyHostToDevice, h->stream));
                CK(mh::launch_ir_start(h->sys, 0.0, iterations, h->stream));
            }
            // warm the captured graph, then time
            if ((rc = capture_iterations(h, prec, ipg, false))) return rc;
            CK(cudaEventRecord(h->ev[0], h->stream));
            // (no restart: the two-kernel iteration, whose launch shape this is about)
            if ((rc = run_krylov(h, prec, ipg, iterations, false))) return rc;
            CK(cudaEventRecord(h->ev[1], h->stream));
            CK(cudaStreamSynchronize(h->stream));
            float ms = 0.f;
            CK(cudaEventElapsedTime(&ms, h->ev[0], h->ev[1]));
            t[k] = 1e3 * ms / iterations;
        }
        // the default solver runs FP32 iterations with an occasional FP64 residual
        const double score = t[1] + 0.05 * t[0];
        if (score < best) {
            best = score;
            best_r = R;
            best32 = t[1];
            best64 = t[0];
        }
    }
    const int targets[2] = {mh::krylov_target_blocks(best_r, 64), mh::krylov_target_blocks(best_r, 32)};
    if ((rc = apply_launch_shape(h, best_r, targets))) return rc;
    if (rows_per_thread) *rows_per_thread = best_r;
    if (us_per_iter) {
        us_per_iter[0] = best32;
        us_per_iter[1] = best64;
    }
    return MH_OK;
}

int mh_set_stream(mh_handle *h, void *cuda_stream) {
    int rc = need_device(h);
    if (rc) return rc;
    CK(cudaStreamSynchronize(h->stream));
    h->stream = cuda_stream ? (cudaStream_t)cuda_stream : h->own_stream;
    return MH_OK;
}

int64_t mh_kernel_launches(const mh_handle *h) { return h ? h->n_launch : 0; }

int mh_learned_set_weights(mh_handle *h, const float *w, int64_t n) {
    int rc = need_device(h);
    if (rc) return rc;
    if (!w || n != mh::kSnParams) {
        h->err = "weights: expected MH_NN_PARAMS floats";
        return MH_ERR_INVALID;
    }
    for (int64_t k = 0; k < n; ++k)
        if (!std::isfinite(w[k])) {
            h->err = "weights: non-finite value";
            return MH_ERR_NONFINITE;
        }
    if ((rc = ensure_learned(h))) return rc;
    h->sn_key_step = -1;  // the next learned solve evaluates the network again
    return nn_upload_weights(h, w);
}

int mh_learned_reset(mh_handle *h) {
    int rc = need_device(h);
    if (rc) return rc;
    if ((rc = ensure_learned(h))) return rc;
    std::vector<float> w;
    nn_initial_params(w, 1);
    h->sn_key_step = -1;
    return nn_upload_weights(h, w.data());
}

int mh_learned_get_weights(const mh_handle *hc, float *w, int64_t n) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    if (!w || n != mh::kSnParams) {
        h->err = "weights: expected MH_NN_PARAMS floats";
        return MH_ERR_INVALID;
    }
    if ((rc = ensure_learned(h))) return rc;
    CK(cudaMemcpyAsync(w, h->nn_w, mh::kSnParams * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return MH_OK;
}

// a training evaluation of one pair given in edge order (see mh_learned_grad)
static int learned_eval_pair(mh_handle *h, const double *r, const double *e, bool refresh, double *loss) {
    int rc = need_device(h);
    if (rc) return rc;
    if (!h->assembled) return MH_ERR_STATE;
    if (!r || !e) return MH_ERR_INVALID;
    if ((rc = ensure_learned(h)) || (rc = ensure_train(h, 1))) return rc;
    const int64_t nr = h->sys.n_rows, ne = h->topo.n_edges();
    std::vector<float> rv(nr, 0.f), ev(nr, 0.f);
    for (int64_t k = 0; k < ne; ++k) {
        const int64_t row = h->hs.edge_row[k];
        rv[row] = (float)r[k];
        ev[row] = (float)e[k];
    }
    if (!h->amg_training || h->tr_hier_epoch != h->matrix_epoch) {
        if ((rc = training_setup(h))) return rc;
        refresh = true;
    }
    CK(cudaMemcpyAsync(h->pair_r, rv.data(), nr * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    CK(cudaMemcpyAsync(h->pair_e, ev.data(), nr * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    // e'S^e in FP32 products, as the loss's numerator
    CK(mh::sn_spmv(h->sys, nullptr, h->pair_e, h->tv[8], h->stream));
    CK(mh::sn_dot(nr, h->pair_e, h->tv[8], h->tdot, h->tdot + 201, h->stream));
    double er = 0.0;
    CK(cudaMemcpyAsync(&er, h->tdot + 201, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    if (!(er > 0.0) || !std::isfinite(er)) {
        h->err = "grad: e'S^e must be positive and finite";
        return MH_ERR_INVALID;
    }
    return train_eval(h, h->pair_r, h->pair_e, er, refresh, loss);
}

int mh_learned_grad(mh_handle *h, const double *r, const double *e, float *grad, double *loss) {
    if (!grad) return MH_ERR_INVALID;
    int rc = learned_eval_pair(h, r, e, true, loss);
    if (rc) return rc;
    CK(cudaMemcpyAsync(grad, h->nn_grad, mh::kSnParams * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    return MH_OK;
}

int mh_learned_grad_weights(mh_handle *h, const double *r, const double *e, int32_t refresh, float *dw, float *w,
                            double *loss) {
    if (!dw && !w && !loss) return MH_ERR_INVALID;
    int rc = learned_eval_pair(h, r, e, refresh != 0, loss);
    if (rc) return rc;
    const int64_t nr = h->sys.n_rows, ne = h->topo.n_edges();
    std::vector<float> a(nr), b(nr);
    CK(cudaMemcpyAsync(a.data(), h->tv[15], nr * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(b.data(), h->sn_w, nr * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    for (int64_t k = 0; k < ne; ++k) {
        if (dw) dw[k] = a[h->hs.edge_row[k]];
        if (w) w[k] = b[h->hs.edge_row[k]];
    }
    return MH_OK;
}

int mh_learned_smoother(mh_handle *h, float *w, int64_t n) {
    int rc = need_device(h);
    if (rc) return rc;
    if (!h->assembled) return MH_ERR_STATE;
    const int64_t nr = h->sys.n_rows, ne = h->topo.n_edges();
    if (!w || n < ne) return MH_ERR_INVALID;
    if ((rc = nn_weights(h))) return rc;
    std::vector<float> a(nr);
    CK(cudaMemcpyAsync(a.data(), h->sn_w, nr * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    for (int64_t k = 0; k < ne; ++k) w[k] = a[h->hs.edge_row[k]];
    h->sn_key_step = -1;
    return MH_OK;
}

int mh_learned_apply(mh_handle *h, const double *r, double *z) {
    int rc = need_device(h);
    if (rc) return rc;
    if (!h->assembled) return MH_ERR_STATE;
    if (!r || !z) return MH_ERR_INVALID;
    if ((rc = ensure_learned(h)) || (rc = ensure_train(h, 1))) return rc;
    if (h->sys.rows_per_thread != 1) {
        const int t[2] = {mh::krylov_target_blocks(1, 64), mh::krylov_target_blocks(1, 32)};
        if ((rc = apply_launch_shape(h, 1, t))) return rc;
    }
    double ms = 0.0;
    if ((rc = prepare_multigrid(h, Pc::Nn, ms))) return rc == MH_FELL_BACK ? MH_ERR_CUDA : rc;
    const int64_t nr = h->sys.n_rows, ne = h->topo.n_edges();
    std::vector<float> rv(nr, 0.f), zv(nr);
    for (int64_t k = 0; k < ne; ++k) rv[h->hs.edge_row[k]] = (float)r[k];
    CK(cudaMemcpyAsync(h->pair_r, rv.data(), nr * sizeof(float), cudaMemcpyHostToDevice, h->stream));
    CK(h->amg.apply(h->pair_r, h->pair_e, nullptr, 0, h->stream));
    h->n_launch += h->amg.kernels_per_apply();
    CK(cudaMemcpyAsync(zv.data(), h->pair_e, nr * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaStreamSynchronize(h->stream));
    for (int64_t k = 0; k < ne; ++k) z[k] = zv[h->hs.edge_row[k]];
    return MH_OK;
}

int mh_amg_info(const mh_handle *hc, int32_t *n_levels, int64_t *rows, int64_t *slots, int32_t cap) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    const mh::Amg &a = h->amg;
    if (n_levels) *n_levels = a.levels();
    for (int l = 0; l < a.levels() && l < cap; ++l) {
        const int64_t real = l == 0 ? a.level(0).A.n : a.level(l - 1).nc;
        if (rows) rows[l] = real;
        if (slots) slots[l] = a.level(l).A.slots;
    }
    return MH_OK;
}

int mh_amg_tail(const mh_handle *hc, int32_t *level, int32_t *cluster_ctas) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    if (level) *level = h->amg.tail_level();
    if (cluster_ctas) *cluster_ctas = h->amg.tail_level() > 0 ? h->amg.tail_cluster() : 0;
    return MH_OK;
}

int mh_amg_coarsest(const mh_handle *hc, int64_t *n, float *inverse) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    if (h->amg.levels() == 0) return MH_ERR_STATE;
    if (n) *n = h->amg.dense_rows();
    if (inverse) CK(h->amg.dense_inverse(inverse, h->stream));
    return MH_OK;
}

int mh_amg_level(const mh_handle *hc, int32_t level, int64_t *n, int64_t *nnz, int32_t *agg, float *weight,
                 int32_t *row_ptr, int32_t *col, float *val) {
    mh_handle *h = const_cast<mh_handle *>(hc);
    int rc = need_device(h);
    if (rc) return rc;
    const mh::Amg &a = h->amg;
    if (level < 0 || level >= a.levels()) return MH_ERR_INVALID;
    const mh::AmgLevel &L = a.level(level);
    const int64_t real = level == 0 ? L.A.n : a.level(level - 1).nc;
    std::vector<int64_t> off(L.A.n_slices + 1);
    std::vector<int32_t> c(L.A.slots);
    std::vector<float> v(L.A.slots);
    CK(cudaMemcpyAsync(off.data(), L.A.slice_off, off.size() * sizeof(int64_t), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(c.data(), L.A.col, c.size() * sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    CK(cudaMemcpyAsync(v.data(), L.A.val, v.size() * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
    if (agg && level + 1 < a.levels())
        CK(cudaMemcpyAsync(agg, L.agg.p, real * sizeof(int32_t), cudaMemcpyDeviceToHost, h->stream));
    if (weight) {
        if (level == 0 && a.fine_weights())
            CK(cudaMemcpyAsync(weight, a.fine_weights(), real * sizeof(float), cudaMemcpyDeviceToHost, h->stream));
        else
            std::fill(weight, weight + real, 1.f);
    }
    CK(cudaStreamSynchronize(h->stream));
    int64_t k = 0;
    if (row_ptr) row_ptr[0] = 0;
    for (int64_t i = 0; i < real; ++i) {
        const int64_t sl = i / mh::kSliceRowsHost, ln = i % mh::kSliceRowsHost;
        const int64_t w = (off[sl + 1] - off[sl]) / mh::kSliceRowsHost;
        auto put = [&](int64_t j) {
            const int64_t slot = off[sl] + j * mh::kSliceRowsHost + ln;
            if (v[slot] == 0.f) return;
            if (col) col[k] = c[slot];
            if (val) val[k] = v[slot];
            ++k;
        };
        // columns ascending: the fine level's rows hold their diagonal in front
        int64_t j = 0;
        if (level == 0) {
            for (j = 1; j < w && c[off[sl] + j * mh::kSliceRowsHost + ln] < i; ++j) put(j);
            put(0);
        }
        for (; j < w; ++j) put(j);
        if (row_ptr) row_ptr[i + 1] = (int32_t)k;
    }
    if (n) *n = real;
    if (nnz) *nnz = k;
    return MH_OK;
}

void mh_learn_opts_default(mh_learn_opts *o) {
    if (!o) return;
    std::memset(o, 0, sizeof(*o));
    o->n_pairs = 12;
    o->epochs = 40;
    o->lr = 2e-3f;
    o->train_bias = 0;
    o->solve_rtol = 1e-9;
    o->seed = 1;
}

int mh_learned_train(mh_handle *h, const mh_learn_opts *opts, mh_learn_stats *stats) {
    int rc = need_device(h);
    if (rc) return rc;
    if (!h->assembled) return MH_ERR_STATE;
    mh_learn_opts o;
    mh_learn_opts_default(&o);
    if (opts) o = *opts;
    mh_learn_stats st;
    std::memset(&st, 0, sizeof(st));
    rc = learned_train_impl(h, o, st);
    if (stats) *stats = st;
    return rc;
}

}  // extern "C"
