// The shared-memory-resident Krylov run (resident.cu): its plan on the host and its launch.
#pragma once
#include <cstdint>
#include <vector>

#include <cuda_runtime.h>

#include "device_system.hpp"

namespace mh {

// Rows per block at least, while the chip has SMs to spare: more blocks cost polls, fewer leave
// rows in line.  6.9k edges: 2.80 us an iteration with 28 blocks (256 rows), 2.71 with 48, 3.11
// with 148; 22k edges: 2.84 with 88 blocks (256 rows), 3.00 with 48, 3.14 with 148.
constexpr int64_t kResidentRows = 256;

// Systems of at most this many rows run in one thread-block cluster: 2.70 us an iteration against
// 2.97 on 49 blocks with 13k rows, 3.43 against 2.79 (FP32 4.01 against 3.36) with 22k.
constexpr int64_t kClusterRows = 14336;

struct ResidentPlan {
    int prec = 64;
    bool cluster = false;             // one cluster of n_blocks blocks instead of a cooperative launch
    int32_t rows_cap = 0;             // rows of the largest block
    int n_blocks = 0, threads = 0;
    int kr = 1;                       // rows per thread
    size_t smem = 0;                  // dynamic shared memory of the largest block
    std::vector<int32_t> blk_slice;   // [n_blocks + 1] first slice of each block
    std::vector<int32_t> halo_off;    // [n_blocks + 1]
    std::vector<int32_t> halo_row;    // rows of other blocks that a block's rows couple to
    std::vector<uint16_t> idx;        // off-diagonal slots: index into the block's own | halo rows
};

struct ResidentDev {
    int32_t *blk_slice = nullptr, *halo_off = nullptr, *halo_row = nullptr;
    uint16_t *idx = nullptr;
    double *part = nullptr;           // 16 doubles per block, zeroed before the first launch
    double *q = nullptr;              // 2 n_rows (value, tag) pairs of the precision, zeroed likewise
    unsigned long long *tag = nullptr;  // 1 before the first launch
    int32_t *err = nullptr;
};

// Plans the run for the current device (prec: 64 or 32); false when the system does not fit.
bool plan_resident(const std::vector<int64_t> &slice_off, const std::vector<int32_t> &col,
                   const std::vector<int32_t> &diag_slot, int prec, ResidentPlan &plan);
// Polls of one value of an exchange (about a second) before a block gives up.
constexpr int kResidentPolls = 1 << 21;
// One Krylov run of a single-instance system, from the state k_cg_init / k_ir_start left, to the
// end of the run; *dev.err != 0 afterwards: an exchange did not complete, x, r, p are worth nothing.
cudaError_t launch_cg_resident(const DevSystem &sys, const ResidentPlan &plan, const ResidentDev &dev, int polls,
                               cudaStream_t s);

}  // namespace mh
