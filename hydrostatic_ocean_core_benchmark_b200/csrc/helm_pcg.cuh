// The on-chip PCG-Jacobi solve of the Helmholtz system (helm_pcg.cu).
#pragma once

#include <cuda_runtime.h>

#include <vector>

namespace oc {

// how a solve's CTAs wait for one another, and what they keep in shared memory
enum { PCG_ONE = 0, PCG_CLUSTER = 1, PCG_GRID = 2 };
enum { PCG_KEEP_ALL = 0, PCG_KEEP_RA = 1, PCG_KEEP_P = 2 };

// Cells up to which one CTA, and up to which one cluster of 16, is the faster
// form: an iteration's work per CTA against what its two barriers cost.
static constexpr int PCG_ONE_CELLS = 2048;
static constexpr int PCG_CLUSTER_CELLS = 65536;

struct PcgParams {
    int nx, ny, n, max_iter, warm;
    double coef, rtol, dx2, dy2;
    const double *mask, *Ku, *Kv, *inv_diag, *rhs;
    double *x, *r, *z, *Ap;  // r and Ap: used when they do not fit shared memory
    int n_leaves, n_slots;
    const int *leaf_start, *leaf_slot;
    double *leafA, *leafB, *leafC;
    int own_max, window;  // cells of the largest range, and of its window of p
    int leaves_max;       // leaves of the range that has most
    int lead;             // window cells before the range (the row below): nx, or 0 for one CTA
    unsigned long long* bar_count;
    int* status;
    long long wait_cycles;
    int *log_iters, *log_conv, *log_count;
    int log_cap;
    __host__ __device__ int window_of(int own) const { return own + 2 * lead; }
};

struct PcgPlan {
    int mode, keep, ncta, own_max, window, leaves_max;
    size_t smem;
};

// a launch for the grid whose NumPy leaves start at `leaves` (n_leaves + 1 offsets);
// false when no form fits (the general solve kernel takes the grid)
bool pcg_plan(const std::vector<int>& leaves, int n_slots, int nx, PcgPlan& plan);
cudaError_t pcg_launch(const PcgPlan& plan, const PcgParams& H, cudaStream_t s);

}  // namespace oc
