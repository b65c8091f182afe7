// Variable-coefficient Helmholtz solver (reference libs/core/solvers_var.py:22-197).
//
// One persistent cooperative kernel runs a whole solve: no host round trip per
// iteration (the reference CUDA backend copies every dot product to the host,
// cfd_exp3d5_cuda.cu:346-352). The stopping test and the CG scalars are
// bit-identical to the reference because every global sum reproduces NumPy's
// pairwise summation: the vector is cut into the same <=128-element leaves,
// each leaf is summed with NumPy's eight interleaved accumulators (eight
// lanes, combined ((0+1)+(2+3))+((4+5)+(6+7)) by shuffles), and the leaf sums
// are folded by the same binary tree. Every CTA folds the tree itself, so all
// CTAs hold the same scalar and take the same branch without another barrier.
//
// Grid-wide barriers are bounded spins: after ~1 s without progress a CTA sets
// OC_ERR_TIMEOUT in the status word and every CTA leaves the solve.
//
// Multigrid fine levels run as shared-memory tiles with a redundant halo (two
// grid barriers per level and V-cycle); levels of at most 32x32 cells run
// inside CTA 0's shared memory.

#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <cmath>
#include <string>
#include <vector>

#include "ocean_b200.h"
#include "grid_barrier.cuh"
#include "helm_common.cuh"
#include "helm_pcg.cuh"
#include "helmholtz.cuh"

namespace oc {

// grids of at most this many cells run their stationary multigrid solve wholly in one CTA.
// MG-preconditioned CG does so up to kCoarseCells only: its vectors stay in global memory,
// and one CTA takes 245 us for 48 x 48 against 205 on every SM.
static constexpr int kOneCtaCells = 2560;
static constexpr int kSolveThreads = 512;  // threads of a solve's CTA
static constexpr int kLeafRow = 136;  // a warp's row of 128 values, the next row in other banks

// ------------------------------------------------------------------ barrier
// the bounded grid barrier of grid_barrier.cuh on the solver's counter and status
__device__ __forceinline__ void grid_sync_begin(const HelmParams& H) { grid_sync_begin(H.status); }

__device__ __forceinline__ bool grid_sync(const HelmParams& H) {
    if (s_grid.ncta == 1) {  // a solve in one CTA waits for nobody
        __syncthreads();
        return true;
    }
    return grid_sync(H.bar_count, H.status, (unsigned)s_grid.ncta, H.wait_cycles);
}

// ------------------------------------------------------------------ level operators
// Gauss-Seidel value of cell e from the neighbours' current x (solvers_var.py:55-69)
__device__ __forceinline__ double gs_at(const HLevel& L, const double* x, const double* b, const Cell& c) {
    const double nb = L.cx * (L.Ku[c.e] * __ldcg(x + c.ie) + L.Ku[c.iw] * __ldcg(x + c.iw)) +
                      L.cy * (L.Kv[c.e] * __ldcg(x + c.jn) + L.Kv[c.js] * __ldcg(x + c.js));
    return L.inv_diag[c.e] * (__ldcg(b + c.e) + nb);
}

__device__ __forceinline__ bool is_colour(const HLevel& L, int e, int colour) {
    const int j = e / L.nx, i = e - j * L.nx;
    return ((i + j) & 1) == colour;
}

// ------------------------------------------------------------------ phases
// Work distribution: `first`/`stride` index the threads taking part (the whole
// grid, or one CTA for the coarse levels).
struct Team {
    int first, stride;
};

__device__ __forceinline__ Team grid_team() {
    Team t;
    t.first = s_grid.cta * blockDim.x + threadIdx.x;
    t.stride = s_grid.ncta * blockDim.x;
    return t;
}


// one colour of a Gauss-Seidel sweep; the cell mask multiply of the sweep end
// is folded into each assignment (identical for wet cells, 0 for dry ones)
__device__ void colour_phase(const HLevel& L, double* x, const double* b, int colour, Team t) {
    for (int e = t.first; e < L.n; e += t.stride) {
        if (!is_colour(L, e, colour)) continue;
        const Cell c = cell_of(L, e);
        x[e] = gs_at(L, x, b, c) * L.mask[e];
    }
}

// ------------------------------------------------------------------ pairwise sums
// element e of a warp's leaf values held as r[e / 32] on lane e mod 32, on every
// lane; e / 32 must be the same on all lanes (the source register is the caller's)
__device__ __forceinline__ double leaf_pick(const double* r, int e) {
    const int q = e >> 5;
    const double x = q == 0 ? r[0] : (q == 1 ? r[1] : (q == 2 ? r[2] : r[3]));
    return __shfl_sync(0xffffffffu, x, e & 31);
}

// NumPy's pairwise sum of one leaf (len <= 128 values) that a warp holds as
// va[q] = element lane + 32 q. The eight interleaved accumulators of NumPy's
// unrolled loop are formed in their sequential order by lanes j = 0..7
// (element 8t + j sits on lane (8t + j) mod 32 in register t / 32, the same
// register on every lane for a given t), folded as
// ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)), and the len mod 8 remaining elements are
// added one by one. Every lane returns the sum.
__device__ __forceinline__ double leaf_sum_warp(const double* va, int len) {
    const int lane8 = threadIdx.x & 7;
    const int m = len >= 8 ? len - (len % 8) : 0;
    double ra = 0.0;
    if (len >= 8) {
        ra = leaf_pick(va, lane8);
        for (int t = 8; t < m; t += 8) ra = ra + leaf_pick(va, t + lane8);
    }
    ra = ra + __shfl_xor_sync(0xffffffffu, ra, 1);
    ra = ra + __shfl_xor_sync(0xffffffffu, ra, 2);
    ra = ra + __shfl_xor_sync(0xffffffffu, ra, 4);
    double a = len >= 8 ? __shfl_sync(0xffffffffu, ra, 0) : 0.0;
    for (int t = m; t < len; ++t) a = a + leaf_pick(va, t);
    return a;
}

// Calls f(e) exactly once per element of level 0, grouped by NumPy's leaves;
// f returns the two values to accumulate. Writes the per-leaf sums. One warp
// per leaf, consecutive leaves on different CTAs; lane l evaluates f for leaf
// elements l, l+32, l+64, l+96 with independent loads.
template <class F>
__device__ void leaf_phase(const HelmParams& H, F f, double* outA, double* outB) {
    const int lane = threadIdx.x & 31;
    const int nwarps = s_grid.ncta * (blockDim.x >> 5);
    const int my = (threadIdx.x >> 5) * s_grid.ncta + s_grid.cta;  // leaf L runs on CTA L mod grid
    for (int L = my; L < H.n_leaves; L += nwarps) {
        const int s = H.leaf_start[L], slot = H.leaf_slot[L];
        const int len = H.leaf_start[L + 1] - s;
        double va[4], vb[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int e = lane + 32 * q;
            double2 v = make_double2(0.0, 0.0);
            if (e < len) v = f(s + e);
            va[q] = v.x;
            vb[q] = v.y;
        }
        const double a = leaf_sum_warp(va, len);
        const double bsum = outB ? leaf_sum_warp(vb, len) : 0.0;
        if (lane == 0) {
            outA[slot] = a;
            if (outB) outB[slot] = bsum;
        }
    }
}

// The fold of the leaf sums for grids with more slots than one CTA folds
// (H.big_fold): the tree is cut below the nodes of at most a block's worth of
// leaves. Each block subtree is folded by one CTA and its root written to
// `broot`; after a grid barrier every CTA folds the top of the tree over the
// block roots. Every addition is the one of the whole-tree fold, in the same
// order, so the result is bit-identical; it costs one more grid barrier. Each
// leaf buffer has its own root buffer, so folds that follow one another without
// a barrier never overwrite roots another CTA is still reading.
__device__ double fold_blocks(const HelmParams& H, const double* leaf, double* broot, double* sm, bool& ok) {
    for (int j = s_grid.cta; j < H.n_blocks; j += s_grid.ncta) {
        const int4 B = H.blocks[j];  // first leaf, leaves, offset of its height starts, heights
        for (int t = threadIdx.x; t < B.y; t += blockDim.x) sm[t] = __ldcg(leaf + B.x + t);
        __syncthreads();
        for (int h = 0; h < B.w; ++h) {
            for (int t = H.bh_start[B.z + h] + threadIdx.x; t < H.bh_start[B.z + h + 1]; t += blockDim.x) {
                const int2 op = H.bops[t];
                sm[op.x] = sm[op.x] + sm[op.y];
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) broot[j] = sm[0];
        __syncthreads();
    }
    ok = grid_sync(H);
    if (!ok) return 0.0;
    for (int t = threadIdx.x; t < H.n_blocks; t += blockDim.x) sm[t] = __ldcg(broot + t);
    __syncthreads();
    for (int h = 0; h < H.top_heights; ++h) {
        for (int t = H.top_hstart[h] + threadIdx.x; t < H.top_hstart[h + 1]; t += blockDim.x) {
            const int2 op = H.top_ops[t];
            sm[op.x] = sm[op.x] + sm[op.y];
        }
        __syncthreads();
    }
    const double r = sm[0];
    __syncthreads();
    return r;
}

// the sum of one of the leaf buffers (leafA, leafB or leafC) in NumPy's order, in
// every CTA (the result is the same everywhere)
__device__ __forceinline__ double fold_sum(const HelmParams& H, const double* leaf, double* sm, bool& ok) {
    if (!H.big_fold) {
        double r[1];
        const double* lv[1] = {leaf};
        slots_fold_any<1>(H.n_slots, lv, sm, r);
        __syncthreads();  // sm is the tiles' next
        return r[0];
    }
    double* broot = leaf == H.leafA ? H.broot : (leaf == H.leafB ? H.broot + H.n_blocks : H.broot + 2 * H.n_blocks);
    return fold_blocks(H, leaf, broot, sm, ok);
}

}  // namespace oc

#include "helm_mg.cuh"

namespace oc {

// ------------------------------------------------------------------ multigrid in one CTA
// The stationary multigrid of a grid of at most kOneCtaCells cells by one CTA (of a
// batched system's share the first; four steps of two members of 48 x 48 x 12 take 12.3 ms
// with the grid-wide form there, 8.2 so): every
// level's coefficients, x and b stay in its shared memory for the solve, all
// barriers are the CTA's, and nothing but the right-hand side and the solution
// crosses global memory. Same operations and sums as the grid-wide form. Squares are
// formed cell by cell into the scratch, in the grid's order, and summed there by
// leaves, four leaves per warp.
__device__ __noinline__ void helm_one_cta(int& iters, int& conv) {
    const HelmParams& H = s_helm;
    const HLevel& L = H.lv[0];
    coarse_tab_init(0, -1);
    const CoarseTab& T = s_ct[0];
    const bool unit = H.unit_mask != 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double* sq = smem_all + s_cres;                    // the squares, after the levels
    double* slots = sq + T.n;                          // leaf sums, then the leaves' starts and slots
    int* start = reinterpret_cast<int*>(slots + H.n_slots);
    int* slot = start + H.n_leaves + 1;
    coarse_coef_load();
    for (int t = threadIdx.x; t < H.n_slots; t += kSolveThreads) slots[t] = 0.0;
    for (int t = threadIdx.x; t <= H.n_leaves; t += kSolveThreads) {
        start[t] = H.leaf_start[t];
        if (t < H.n_leaves) slot[t] = H.leaf_slot[t];
    }
    for (int e = threadIdx.x; e < T.n; e += kSolveThreads) {
        const int j = fast_div(e, T.nmag), o = coarse_pos(T, e - j * T.nx, j);
        const double r = H.rhs[e] * __ldg(L.mask + e);
        smem_all[T.b + o] = r;
        smem_all[T.x + o] = H.warm ? L.x[e] : 0.0;
        sq[e] = r * r;
    }
    cpa_wait_all();
    __syncthreads();
    // the square root of the squares' sum in NumPy's pairwise order
    auto norm = [&]() {
        for (int l0 = 4 * warp; l0 < H.n_leaves; l0 += 4 * (kSolveThreads / 32)) {
            const int l = l0 + (lane >> 3), j = lane & 7;
            const int st = l < H.n_leaves ? start[l] : 0, len = l < H.n_leaves ? start[l + 1] - st : 0, m = len & ~7;
            double acc = 0.0;
            if (m) {
                acc = sq[st + j];
#pragma unroll 4
                for (int t = 8; t < m; t += 8) acc = acc + sq[st + t + j];
            }
            acc = acc + __shfl_xor_sync(0xffffffffu, acc, 1);
            acc = acc + __shfl_xor_sync(0xffffffffu, acc, 2);
            acc = acc + __shfl_xor_sync(0xffffffffu, acc, 4);
            for (int t = m; t < len; ++t) acc = acc + sq[st + t];
            if (l < H.n_leaves && j == 0) slots[slot[l]] = acc;
        }
        __syncthreads();
        const double x = H.n_slots == 32 ? warp_tree<1>(slots, false) : warp_tree<2>(slots, false);
        return sqrt(__shfl_sync(0xffffffffu, x, 0));
    };
    const double norm_b = norm();
    iters = 0;
    conv = 1;
    if (norm_b != 0.0) {
        const double tol = H.rtol * norm_b;
        conv = 0;
        for (int it = 1; it <= H.max_iter; ++it) {
            coarse_cycle();
            iters = it;
            // the residual of the stopping test is not masked (solvers_var.py:170-179)
            if (T.even) {
                for (int f = threadIdx.x; f < T.n; f += kSolveThreads) {
                    const int p = f >= T.nh, q = f - p * T.nh;
                    const double d = coarse_residual(T, H.coef, unit, p, q, false);
                    const int j = fast_div(q, T.hmag);
                    sq[j * T.nx + 2 * (q - j * T.hx) + ((p + j) & 1)] = d * d;
                }
            } else {
                const double *x = smem_all + T.x, *mk = smem_all + T.m;
                for (int e = threadIdx.x; e < T.n; e += kSolveThreads) {
                    const Cell c = cell_of(L, e);
                    const double m = mk[e], xm = x[e] * m;
                    const double fx = smem_all[T.ku + e] * (x[c.ie] * mk[c.ie] - xm);
                    const double fxw = smem_all[T.ku + c.iw] * (xm - x[c.iw] * mk[c.iw]);
                    const double fy = smem_all[T.kv + e] * (x[c.jn] * mk[c.jn] - xm);
                    const double fys = smem_all[T.kv + c.js] * (xm - x[c.js] * mk[c.js]);
                    const double lap = (fx - fxw) / T.dx2 + (fy - fys) / T.dy2;
                    const double d = smem_all[T.b + e] - ((xm - H.coef * lap) * m + xm * (1.0 - m));
                    sq[e] = d * d;
                }
            }
            __syncthreads();
            const double res = norm();
            if (res <= tol) {
                conv = 1;
                break;
            }
        }
    }
    for (int e = threadIdx.x; e < T.n; e += kSolveThreads) {
        const int j = fast_div(e, T.nmag);
        L.x[e] = smem_all[T.x + coarse_pos(T, e - j * T.nx, j)];
    }
}

// the leaf sums of the squared residual of x (not masked, as the stopping test takes it)
// into leafA, beside level 0's down phase: on the CTAs without a tile when each of
// their warps then has at most one leaf, else on all, those with the fewest tiles first
__device__ __noinline__ void residual_leaves(const double* x) {
    const HelmParams& H = s_helm;
    const HLevel& L0 = H.lv[0];
    // with CTAs to spare the tiles sit on the last ones
    const int idle = s_grid.ncta - level_tiles(L0), warps = kSolveThreads / 32;
    const bool apart = idle > 0 && idle * warps >= H.n_leaves;
    const int rank = s_grid.cta;
    const int n = apart ? idle : s_grid.ncta;
    if (rank >= n) return;
    const int lane = threadIdx.x & 31;
    for (int L = (threadIdx.x >> 5) * n + rank; L < H.n_leaves; L += n * warps) {
        const int s = H.leaf_start[L], len = H.leaf_start[L + 1] - s, slot = H.leaf_slot[L];
        double v[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            v[q] = 0.0;
            if (lane + 32 * q < len) {
                const int e = s + lane + 32 * q;
                const double d = __ldcg(L0.b + e) - apply_at(L0, H.coef, x, cell_of(L0, e));
                v[q] = d * d;
            }
        }
        const double a = leaf_sum_warp(v, len);
        if (lane == 0) H.leafA[slot] = a;
    }
}

// ------------------------------------------------------------------ the solve kernel
// A whole solve on the CTAs s_grid names (set by the kernel, followed by a CTA
// barrier, before the call).
__device__ __forceinline__ void solve_log(const HelmParams& H, bool ok, int iters, int conv) {
    if (s_grid.cta != 0 || threadIdx.x != 0) return;
    const int idx = *H.log_count;
    if (idx < H.log_cap) {
        H.log_iters[idx] = ok ? iters : -1;
        H.log_conv[idx] = ok ? conv : 0;
    }
    *H.log_count = idx + 1;
}

// MG: with the V-cycle; without it the multigrid kinds are not reached.
template <bool MG>
__device__ __forceinline__ void helm_solve_body() {
    const HelmParams& H = s_helm;
    if constexpr (MG) {
        if (H.one_cta) {
            if (s_grid.cta != 0) return;  // of a batched system's share the first CTA
            int its, cv;
            helm_one_cta(its, cv);
            solve_log(H, true, its, cv);
            return;
        }
    }
    // with H.persist0 the first 4 SN doubles (6 with its x and b) hold level 0's tile for the
    // whole solve; every other use of shared memory works above them
    const int persist = MG && H.persist0 ? 0 : -1;
    const int smo = MG && H.persist0 ? (H.keep_x0 ? 6 : 4) * TileWide::SN : 0;
    double* sm = smem_all + smo;
    const HLevel& L0 = H.lv[0];
    const double* rhs = H.rhs;
    double* x = L0.x;
    double* b0 = L0.b;
    bool ok = true;
    int iters = 0, conv = 1;
    grid_sync_begin(H);

    // norm of the masked right-hand side (solvers_var.py:163-168)
    leaf_phase(H,
               [&](int e) {
                   const double r = rhs[e] * L0.mask[e];
                   b0[e] = r;
                   // the CG residual of the starting iterate: b, or b - A x with a warm start
                   if (H.kind <= HK_PCG_RBGS || H.kind == HK_PCG_MG)
                       H.r[e] = H.warm ? r - apply_at(L0, H.coef, x, cell_of(L0, e)) : r;
                   if (!H.warm) x[e] = 0.0;
                   return make_double2(r * r, 0.0);
               },
               H.leafA, nullptr);
    ok = grid_sync(H);
    const double norm_b = ok ? sqrt(fold_sum(H, H.leafA, sm, ok)) : 0.0;
    if constexpr (MG) {
        if (persist >= 0) persist_level0(smo, persist);  // the coefficients are fixed during the solve
        if (s_grid.cta == 0 && H.coarse_from < H.n_levels) {
            coarse_tab_init(smo, coarse_coef_at(H, smo, persist));
            if (s_coarse_held) {
                coarse_coef_load();
                cpa_wait_all();
                __syncthreads();
            }
        }
    }
    if (!ok || norm_b == 0.0) goto done;
    {
        const double tol = H.rtol * norm_b;
        if (H.kind == HK_RBGS || (MG && H.kind == HK_MULTIGRID)) {
            // stationary iteration with the true residual (solvers_var.py:170-179)
            conv = 0;
            double* xc = x;  // the level-0 buffer holding the current iterate
            // Where the up phase does not form the residual's leaf sums, they are formed
            // beside the next cycle's first phase, on the CTAs that have no tile in it if
            // they are enough: a grid barrier and a pass of their own less per cycle, for
            // one phase that the last cycle runs in vain.
            const bool piped = MG && H.kind == HK_MULTIGRID && !H.fused_res && H.coarse_from > 0 && H.n_levels > 1;
            for (int it = 1; it <= H.max_iter && ok; ++it) {
                if (MG && H.kind == HK_MULTIGRID) {
                    if constexpr (MG) {
                        // the previous iterate's residual and its test, beside this cycle's first phase
                        const double* xp = xc;
                        xc = vcycle_tiled(H, xc, xc == H.lv[0].x ? H.lv[0].x2 : H.lv[0].x, smo, persist, ok,
                                          [&]() { if (piped && it > 1) residual_leaves(xp); },
                                          [&]() {
                                              if (!piped || it == 1) return false;
                                              iters = it - 1;
                                              conv = sqrt(fold_sum(H, H.leafA, sm, ok)) <= tol ? 1 : 0;
                                              return conv != 0 || !ok;
                                          });
                        if (conv) break;
                    }
                } else {
                    colour_phase(L0, x, b0, 0, grid_team());
                    ok = grid_sync(H);
                    if (!ok) break;
                    colour_phase(L0, x, b0, 1, grid_team());
                    ok = grid_sync(H);
                }
                if (!ok) break;
                if (piped && it < H.max_iter) continue;
                // the true residual's leaf sums: formed by the last up phase when
                // level 0's tiles are NumPy's leaves, else by a pass of their own
                if (!(MG && H.kind == HK_MULTIGRID && H.fused_res)) {
                    const double* xr = xc;
                    leaf_phase(H,
                               [&](int e) {
                                   const double d = __ldcg(b0 + e) - apply_at(L0, H.coef, xr, cell_of(L0, e));
                                   return make_double2(d * d, 0.0);
                               },
                               H.leafA, nullptr);
                    ok = grid_sync(H);
                    if (!ok) break;
                }
                iters = it;
                const double res = sqrt(fold_sum(H, H.leafA, sm, ok));
                if (!ok) break;
                if (res <= tol) {
                    conv = 1;
                    break;
                }
            }
            if (ok && xc != x) {
                for (int e = grid_team().first; e < L0.n; e += grid_team().stride) x[e] = __ldcg(xc + e);
            }
        } else {
            // preconditioned CG (solvers_var.py:181-197). A fold reads its leaf
            // sums after a grid barrier, and a leaf phase that follows a fold with
            // no barrier between them writes a different buffer: a CTA that leaves
            // its fold early must not overwrite sums another CTA is still reading.
            // <r,z> at the start: leafB (leafA holds |b|); <p,Ap>: leafC; <r,r>
            // and <r,z> of the update: leafA and leafB, read last before the
            // barrier that ends the previous iteration.
            double* r = H.r;
            double* z = H.z;
            double* p = H.p;
            double* Ap = H.Ap;
            const bool jac = H.kind == HK_PCG_JACOBI;
            // z = M^-1 r
            auto precondition = [&](bool& okp) {
                if (jac) return;
                if constexpr (MG) {
                    if (H.kind == HK_PCG_MG) {
                        // one V(2,2) cycle on level 0's rhs r from a zero iterate (symmetric:
                        // red-black pre-smoothing, black-red post-smoothing)
                        for (int e = grid_team().first; e < L0.n; e += grid_team().stride) {
                            b0[e] = __ldcg(r + e);
                            z[e] = 0.0;
                        }
                        okp = grid_sync(H);
                        if (!okp) return;
                        double* zr = vcycle_tiled(H, z, L0.x2, smo, persist, okp, []() {}, []() { return false; });
                        if (!okp || zr == z) return;
                        for (int e = grid_team().first; e < L0.n; e += grid_team().stride) z[e] = __ldcg(zr + e);
                        okp = grid_sync(H);
                        return;
                    }
                }
                for (int e = grid_team().first; e < L0.n; e += grid_team().stride) z[e] = 0.0;
                okp = grid_sync(H);
                if (!okp) return;
                for (int h = 0; h < 4 && okp; ++h) {
                    const int colour = (h == 0 || h == 3) ? 0 : 1;
                    colour_phase(L0, z, r, colour, grid_team());
                    okp = grid_sync(H);
                }
            };
            precondition(ok);
            if (!ok) goto done;
            leaf_phase(H,
                       [&](int e) {
                           const double re = __ldcg(r + e);
                           const double ze = jac ? L0.inv_diag[e] * re : __ldcg(z + e);
                           if (jac) z[e] = ze;
                           p[e] = ze;
                           return make_double2(re * ze, 0.0);
                       },
                       H.leafB, nullptr);
            ok = grid_sync(H);
            if (!ok) goto done;
            double rz = fold_sum(H, H.leafB, sm, ok);
            if (!ok) goto done;
            conv = 0;
            for (int it = 1; it <= H.max_iter; ++it) {
                leaf_phase(H,
                           [&](int e) {
                               const double a = apply_at(L0, H.coef, p, cell_of(L0, e));
                               Ap[e] = a;
                               return make_double2(__ldcg(p + e) * a, 0.0);
                           },
                           H.leafC, nullptr);
                ok = grid_sync(H);
                if (!ok) break;
                const double alpha = rz / fold_sum(H, H.leafC, sm, ok);
                if (!ok) break;
                leaf_phase(H,
                           [&](int e) {
                               const double pe = __ldcg(p + e);
                               const double ae = __ldcg(Ap + e);
                               const double xe = __ldcg(x + e) + alpha * pe;
                               const double re = __ldcg(r + e) - alpha * ae;
                               x[e] = xe;
                               r[e] = re;
                               double ze = 0.0;
                               if (jac) {
                                   ze = L0.inv_diag[e] * re;
                                   z[e] = ze;
                               }
                               return make_double2(re * re, re * ze);
                           },
                           H.leafA, H.leafB);
                ok = grid_sync(H);
                if (!ok) break;
                iters = it;
                const double res = sqrt(fold_sum(H, H.leafA, sm, ok));
                if (!ok) break;
                if (res <= tol) {
                    conv = 1;
                    break;
                }
                if (!jac) {
                    precondition(ok);
                    if (!ok) break;
                    leaf_phase(H,
                               [&](int e) {
                                   const double re = __ldcg(r + e);
                                   return make_double2(re * __ldcg(z + e), 0.0);
                               },
                               H.leafB, nullptr);
                    ok = grid_sync(H);
                    if (!ok) break;
                }
                const double rz_new = fold_sum(H, H.leafB, sm, ok);
                if (!ok) break;
                const double beta = rz_new / rz;
                for (int e = grid_team().first; e < L0.n; e += grid_team().stride)
                    p[e] = __ldcg(z + e) + beta * __ldcg(p + e);
                ok = grid_sync(H);
                if (!ok) break;
                rz = rz_new;
            }
        }
    }
done:
    grid_sync_end(H.bar_count, s_grid.cta == 0);
    solve_log(H, ok, iters, conv);
}

// The parameters are read through a reference throughout the solve: a copy in
// shared memory, made once per CTA (a reference to the kernel parameter itself
// would give every thread a copy of its own in local memory).
// One kernel for the multigrid kinds and one for the others, which in one kernel with the
// V-cycle spill (128 registers and 328 bytes of stack; 110 and none apart). us a solve
// together and apart: PCG-RBGS 48 x 48 294 and 279, 1000 x 720 1019 and 979; RBGS 128 x 96
// 237 and 229; four steps of eight PCG-Jacobi members, batched, 34.3 and 32.4
// ms. Without the bound of one CTA per SM the compiler gives the second one 64
// registers and spills, and two CTAs per SM wait for one another: PCG-RBGS 128 x 96 321
// against 297.
template <bool MG>
__global__ void __launch_bounds__(512, MG ? 0 : 1) k_helm_solve(HelmParams H) {
    if (threadIdx.x == 0) s_grid = SolveGrid{(int)blockIdx.x, (int)gridDim.x};
    const int* src = reinterpret_cast<const int*>(&H);
    int* dst = reinterpret_cast<int*>(&s_helm);
    for (int t = threadIdx.x; t < (int)(sizeof(HelmParams) / sizeof(int)); t += blockDim.x) dst[t] = src[t];
    __syncthreads();
    helm_solve_body<MG>();
}

// Several systems in one cooperative launch: system m runs on CTAs
// [cta_start[m], cta_start[m + 1]) with its own parameters (copied into shared
// memory), its own barrier counter, status word and solve log; the systems
// never wait on one another.
// MG: at least one of them is of a multigrid kind.
template <bool MG>
__global__ void __launch_bounds__(512, MG ? 0 : 1) k_helm_solve_batched(const HelmParams* __restrict__ systems,
                                                            const int* __restrict__ cta_start, int n) {
    __shared__ int s_m;
    if (threadIdx.x == 0) {
        int m = 0;
        while (m + 1 < n && (int)blockIdx.x >= cta_start[m + 1]) ++m;
        s_m = m;
        s_grid = SolveGrid{(int)blockIdx.x - cta_start[m], cta_start[m + 1] - cta_start[m]};
    }
    __syncthreads();
    const int* src = reinterpret_cast<const int*>(systems + s_m);
    int* dst = reinterpret_cast<int*>(&s_helm);
    for (int t = threadIdx.x; t < (int)(sizeof(HelmParams) / sizeof(int)); t += blockDim.x) dst[t] = src[t];
    __syncthreads();
    helm_solve_body<MG>();
}

// ------------------------------------------------------------------ level rebuild
// coarse face coefficients (solvers_var.py:118-123) and inverse diagonal
// (solvers_var.py:39-45) of level `L` from the finer level `F`
__global__ void k_helm_level(HLevel F, HLevel L, int coarse, int unit_mask) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= L.n) return;
    const int J = e / L.nx, I = e - J * L.nx;
    const int Iw = I == 0 ? L.nx - 1 : I - 1, Js = J == 0 ? L.ny - 1 : J - 1;
    double ku, kuw, kv, kvs;
    if (coarse) {
        auto cku = [&](int jj, int ii) {
            return 0.5 * (F.Ku[(2 * jj) * F.nx + 2 * ii + 1] + F.Ku[(2 * jj + 1) * F.nx + 2 * ii + 1]);
        };
        auto ckv = [&](int jj, int ii) {
            return 0.5 * (F.Kv[(2 * jj + 1) * F.nx + 2 * ii] + F.Kv[(2 * jj + 1) * F.nx + 2 * ii + 1]);
        };
        ku = cku(J, I);
        kuw = cku(J, Iw);
        kv = ckv(J, I);
        kvs = ckv(Js, I);
        L.Ku[e] = ku;
        L.Kv[e] = kv;
    } else {
        ku = L.Ku[e];
        kuw = L.Ku[J * L.nx + Iw];
        kv = L.Kv[e];
        kvs = L.Kv[Js * L.nx + I];
    }
    const double d = 1.0 + L.cx * (ku + kuw) + L.cy * (kv + kvs);
    const double inv = 1.0 / (L.mask[e] > 0.0 ? d : 1.0);
    L.inv_diag[e] = inv;
    if (L.idm != L.inv_diag) L.idm[e] = unit_mask ? inv * L.mask[e] : inv;
}

// ------------------------------------------------------------------ host side
// NumPy's pairwise summation tree of n contiguous elements
// (numpy/core/src/umath/loops_utils.h.src, pairwise_sum: leaves of <= 128
// elements, split at n/2 rounded down to a multiple of 8)
struct PwNode {
    int lo, height;
};

// The tree embedded in a perfect one: where each leaf starts and its slot, in order, under a
// node of height `height` (2^height slots) whose first slot is `slot`. A leaf
// above height 0 takes the first slot of its subtree.
static int pairwise_height(long n) {
    if (n <= 128) return 0;
    long h = n / 2;
    h -= h % 8;
    return std::max(pairwise_height(h), pairwise_height(n - h)) + 1;
}

static void pairwise_slots(long start, long n, int height, int slot, std::vector<int>& leaves, std::vector<int>& slots) {
    if (n <= 128) {
        leaves.push_back((int)start);
        slots.push_back(slot);
        return;
    }
    long h = n / 2;
    h -= h % 8;
    pairwise_slots(start, h, height - 1, slot, leaves, slots);
    pairwise_slots(start + h, n - h, height - 1, slot + (1 << (height - 1)), leaves, slots);
}

static PwNode pairwise_build(long start, long n, std::vector<int>& leaves,
                             std::vector<std::vector<int2>>& by_height) {
    if (n <= 128) {
        leaves.push_back((int)start);
        return {(int)leaves.size() - 1, 0};
    }
    long h = n / 2;
    h -= h % 8;
    const PwNode a = pairwise_build(start, h, leaves, by_height);
    const PwNode b = pairwise_build(start + h, n - h, leaves, by_height);
    const int height = std::max(a.height, b.height) + 1;
    if ((int)by_height.size() < height) by_height.resize(height);
    by_height[height - 1].push_back(make_int2(a.lo, b.lo));
    return {a.lo, height};
}

// leaves of NumPy's pairwise tree over n contiguous elements
static long pairwise_leaves(long n) {
    if (n <= 128) return 1;
    long h = n / 2;
    h -= h % 8;
    return pairwise_leaves(h) + pairwise_leaves(n - h);
}

// The two-level form of the same tree: nodes of at most `block_leaves` leaves
// become blocks, each with its own plan (leaf indices relative to its first
// leaf; `hstart` gets heights + 1 offsets into `bops` per block), and the nodes
// above them form the top plan over the block indices. `leaves` receives every
// leaf in order, as pairwise_build gives them.
struct TwoLevelPlan {
    std::vector<int> leaves;
    std::vector<int4> blocks;
    std::vector<int2> bops;
    std::vector<int> bh_start;
    std::vector<std::vector<int2>> top_by_height;
};

static PwNode pairwise_build_two_level(long start, long n, long block_leaves, TwoLevelPlan& T) {
    if (pairwise_leaves(n) <= block_leaves) {
        std::vector<int> lv;
        std::vector<std::vector<int2>> byh;
        pairwise_build(start, n, lv, byh);
        const int4 b = make_int4((int)T.leaves.size(), (int)lv.size(), (int)T.bh_start.size(), (int)byh.size());
        T.leaves.insert(T.leaves.end(), lv.begin(), lv.end());
        for (const auto& ops : byh) {
            T.bh_start.push_back((int)T.bops.size());
            T.bops.insert(T.bops.end(), ops.begin(), ops.end());
        }
        T.bh_start.push_back((int)T.bops.size());
        T.blocks.push_back(b);
        return {(int)T.blocks.size() - 1, 0};
    }
    long h = n / 2;
    h -= h % 8;
    const PwNode a = pairwise_build_two_level(start, h, block_leaves, T);
    const PwNode b = pairwise_build_two_level(start + h, n - h, block_leaves, T);
    const int height = std::max(a.height, b.height) + 1;
    if ((int)T.top_by_height.size() < height) T.top_by_height.resize(height);
    T.top_by_height[height - 1].push_back(make_int2(a.lo, b.lo));
    return {a.lo, height};
}

// leaf sums beyond which the fold runs in two levels (their doubles would not
// fit one CTA's shared memory beside the rest), and the leaves of one block
static constexpr long kFoldOneLevelLeaves = 16384;
static constexpr long kFoldBlockLeaves = 8192;

// Raises a solve kernel's shared-memory allowance on device `dev` to `smem` dynamic bytes.
// The allowance belongs to the kernel on the device, not to a solver, and only ever
// grows, so the solvers of other grids keep launching. What a kernel may have without it
// is 48 KB less its static shared memory, so every size asks.
static cudaError_t allow_smem(const void* kernel, size_t smem, int dev) {
    static std::mutex mu;
    static std::map<std::pair<int, const void*>, size_t> allowance;
    std::lock_guard<std::mutex> lock(mu);
    size_t& a = allowance[{dev, kernel}];
    if (smem <= a) return cudaSuccess;
    const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) a = smem;
    return e;
}

void* HelmSolver::dalloc(size_t nbytes) {
    void* p = nullptr;
    if (cudaMalloc(&p, nbytes) != cudaSuccess) return nullptr;
    cudaMemset(p, 0, nbytes);
    allocs_.push_back(p);
    bytes_ += nbytes;
    return p;
}

HelmSolver::~HelmSolver() {
    delete refined_;
    for (void* p : allocs_) cudaFree(p);
}

int HelmSolver::init(int nx, int ny, double dx0, double dy0, double coef, int kind, double rtol,
                     int max_iter, const double* mask_host, double* Ku, double* Kv, int log_cap,
                     int* status, std::string& err) {
    HelmParams& H = hp_;
    // the refined solver keeps this solver's log, counters and level-0 arrays
    // (built as for PCG-Jacobi) and runs its solves itself
    const bool refined = kind == HK_REFINED;
    if (refined) kind = HK_PCG_JACOBI;
    H.kind = kind;
    H.coef = coef;
    H.rtol = rtol;
    H.max_iter = max_iter;
    H.status = status;
    H.unit_mask = 1;
    for (size_t c = 0; c < (size_t)nx * ny && H.unit_mask; ++c) H.unit_mask = mask_host[c] == 0.0 || mask_host[c] == 1.0;
    // level geometry and masks
    std::vector<std::vector<double>> masks;
    masks.push_back(std::vector<double>(mask_host, mask_host + (size_t)nx * ny));
    int lnx = nx, lny = ny;
    std::vector<std::pair<int, int>> dims{{nx, ny}};
    const bool mg_levels = kind == HK_MULTIGRID || kind == HK_PCG_MG;
    if (mg_levels) {
        while (lnx % 2 == 0 && lny % 2 == 0 && lnx / 2 >= 8 && lny / 2 >= 8 &&
               (int)dims.size() < OC_MAX_LEVELS) {
            const int cnx = lnx / 2, cny = lny / 2;
            const std::vector<double>& fm = masks.back();
            std::vector<double> cm((size_t)cnx * cny);
            for (int J = 0; J < cny; ++J)
                for (int I = 0; I < cnx; ++I) {
                    const double a = fm[(size_t)(2 * J) * lnx + 2 * I], b = fm[(size_t)(2 * J) * lnx + 2 * I + 1];
                    const double c = fm[(size_t)(2 * J + 1) * lnx + 2 * I], d = fm[(size_t)(2 * J + 1) * lnx + 2 * I + 1];
                    cm[(size_t)J * cnx + I] = std::max(std::max(std::max(a, b), c), d);
                }
            masks.push_back(cm);
            dims.push_back({cnx, cny});
            lnx = cnx;
            lny = cny;
        }
    }
    H.n_levels = (int)dims.size();
    H.coarse_from = H.n_levels;
    for (int l = 0; l < H.n_levels; ++l) {
        HLevel& L = H.lv[l];
        L.nx = dims[l].first;
        L.ny = dims[l].second;
        L.n = L.nx * L.ny;
        // coarse level l spans the same length with nx / 2^l cells: Lx / (nx / 2^l)
        // is exactly (Lx / nx) * 2^l, the reference's CGrid spacing of that level
        const double dx = std::ldexp(dx0, l), dy = std::ldexp(dy0, l);
        L.dx2 = std::pow(dx, 2.0);
        L.dy2 = std::pow(dy, 2.0);
        L.cx = coef * (1.0 / std::pow(dx, 2.0));
        L.cy = coef * (1.0 / std::pow(dy, 2.0));
        double* m = (double*)dalloc(sizeof(double) * L.n);
        if (!m) {
            err = "cudaMalloc failed (Helmholtz levels)";
            return OC_ERR_CUDA;
        }
        cudaMemcpy(m, masks[l].data(), sizeof(double) * L.n, cudaMemcpyHostToDevice);
        L.mask = m;
        L.inv_diag = (double*)dalloc(sizeof(double) * L.n);
        L.idm = mg_levels ? (double*)dalloc(sizeof(double) * L.n) : L.inv_diag;
        L.b = (double*)dalloc(sizeof(double) * L.n);
        L.x2 = (double*)dalloc(sizeof(double) * L.n);
        if (l == 0) {
            L.Ku = Ku;
            L.Kv = Kv;
            L.x = nullptr;  // set per solve
        } else {
            L.Ku = (double*)dalloc(sizeof(double) * L.n);
            L.Kv = (double*)dalloc(sizeof(double) * L.n);
            L.x = (double*)dalloc(sizeof(double) * L.n);
        }
        if (!L.inv_diag || !L.idm || !L.b || !L.x2 || (l > 0 && (!L.Ku || !L.Kv || !L.x))) {
            err = "cudaMalloc failed (Helmholtz levels)";
            return OC_ERR_CUDA;
        }
        if (L.n <= (l == 0 && kind == HK_MULTIGRID ? kOneCtaCells : kCoarseCells) && H.coarse_from == H.n_levels) H.coarse_from = l;
    }
    const size_t n = (size_t)nx * ny;
    H.r = (double*)dalloc(sizeof(double) * n);
    H.z = (double*)dalloc(sizeof(double) * n);
    H.p = (double*)dalloc(sizeof(double) * n);
    H.Ap = (double*)dalloc(sizeof(double) * n);
    // pairwise plan (two-level for grids whose leaf sums exceed shared memory)
    std::vector<int> leaves, slots;
    TwoLevelPlan two;
    H.big_fold = pairwise_leaves((long)n) > kFoldOneLevelLeaves ? 1 : 0;
    if (H.big_fold) {
        pairwise_build_two_level(0, (long)n, kFoldBlockLeaves, two);
        leaves = two.leaves;
        // the two-level fold reads the leaves in order
        for (int q = 0; q < (int)leaves.size(); ++q) slots.push_back(q);
        H.n_slots = (int)slots.size();
    } else {
        // the leaves' slots in the perfect tree (at least one warp's 32)
        const int height = pairwise_height((long)n);
        pairwise_slots(0, (long)n, height, 0, leaves, slots);
        H.n_slots = std::max(32, 1 << height);
    }
    leaves.push_back((int)n);
    H.n_leaves = (int)leaves.size() - 1;
    int* d_leaves = (int*)dalloc(sizeof(int) * leaves.size());
    int* d_slots = (int*)dalloc(sizeof(int) * slots.size());
    H.leafA = (double*)dalloc(sizeof(double) * H.n_slots);  // zeroed: slots without a leaf stay 0
    H.leafB = (double*)dalloc(sizeof(double) * H.n_slots);
    H.leafC = (double*)dalloc(sizeof(double) * H.n_slots);
    unsigned long long* bar = (unsigned long long*)dalloc(sizeof(unsigned long long));
    H.log_cap = log_cap;
    H.log_iters = (int*)dalloc(sizeof(int) * log_cap);
    H.log_conv = (int*)dalloc(sizeof(int) * log_cap);
    H.log_count = (int*)dalloc(sizeof(int));
    if (!H.r || !H.z || !H.p || !H.Ap || !d_leaves || !d_slots || !H.leafA || !H.leafB || !H.leafC ||
        !bar || !H.log_iters || !H.log_conv || !H.log_count) {
        err = "cudaMalloc failed (Helmholtz work)";
        return OC_ERR_CUDA;
    }
    cudaMemcpy(d_leaves, leaves.data(), sizeof(int) * leaves.size(), cudaMemcpyHostToDevice);
    cudaMemcpy(d_slots, slots.data(), sizeof(int) * slots.size(), cudaMemcpyHostToDevice);
    H.leaf_start = d_leaves;
    H.leaf_slot = d_slots;
    H.bar_count = bar;
    H.wait_cycles = kBarrierCycles;
    size_t fold_doubles = 32;  // shared memory the fold needs
    if (H.big_fold) {
        H.n_blocks = (int)two.blocks.size();
        std::vector<int> top_hstart{0};
        std::vector<int2> top_ops;
        for (auto& v : two.top_by_height) {
            top_ops.insert(top_ops.end(), v.begin(), v.end());
            top_hstart.push_back((int)top_ops.size());
        }
        H.top_heights = (int)two.top_by_height.size();
        int4* d_blocks = (int4*)dalloc(sizeof(int4) * two.blocks.size());
        int2* d_bops = (int2*)dalloc(sizeof(int2) * std::max<size_t>(1, two.bops.size()));
        int* d_bh = (int*)dalloc(sizeof(int) * two.bh_start.size());
        int2* d_top = (int2*)dalloc(sizeof(int2) * std::max<size_t>(1, top_ops.size()));
        int* d_top_h = (int*)dalloc(sizeof(int) * top_hstart.size());
        H.broot = (double*)dalloc(sizeof(double) * 3 * (size_t)H.n_blocks);
        if (!d_blocks || !d_bops || !d_bh || !d_top || !d_top_h || !H.broot) {
            err = "cudaMalloc failed (Helmholtz reduction plan)";
            return OC_ERR_CUDA;
        }
        cudaMemcpy(d_blocks, two.blocks.data(), sizeof(int4) * two.blocks.size(), cudaMemcpyHostToDevice);
        if (!two.bops.empty())
            cudaMemcpy(d_bops, two.bops.data(), sizeof(int2) * two.bops.size(), cudaMemcpyHostToDevice);
        cudaMemcpy(d_bh, two.bh_start.data(), sizeof(int) * two.bh_start.size(), cudaMemcpyHostToDevice);
        if (!top_ops.empty())
            cudaMemcpy(d_top, top_ops.data(), sizeof(int2) * top_ops.size(), cudaMemcpyHostToDevice);
        cudaMemcpy(d_top_h, top_hstart.data(), sizeof(int) * top_hstart.size(), cudaMemcpyHostToDevice);
        H.blocks = d_blocks;
        H.bops = d_bops;
        H.bh_start = d_bh;
        H.top_ops = d_top;
        H.top_hstart = d_top_h;
        fold_doubles = (size_t)H.n_blocks;
        for (const int4& b : two.blocks) fold_doubles = std::max(fold_doubles, (size_t)b.y);
    }
    // co-resident grid for the cooperative launch
    int dev = 0, sms = 0, coop = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (!coop) {
        err = "device does not support cooperative launches";
        return OC_ERR_UNSUPPORTED;
    }
    size_t coarse_cells = 0;
    for (int l = H.coarse_from; l < H.n_levels; ++l) coarse_cells += (size_t)H.lv[l].n;
    // Level 0 of a grid whose 32 x 32 tiles need more than one round over the SMs
    // runs 128 x 16 tiles instead. When NumPy's leaves are then exactly the tiles'
    // 128-cell rows, the last up phase forms the residual's leaf sums itself.
    const bool grid_levels = mg_levels && H.n_levels >= 2 && H.coarse_from >= 1;
    const long long tiles32 = (long long)((nx + 31) / 32) * ((ny + 31) / 32);
    H.wide0 = (grid_levels && nx % TileWide::TX == 0 && tiles32 > sms) ? 1 : 0;
    // every other grid level takes the smallest tile whose count fits one round
    // over the SMs: the phases are latency-bound, so less work per CTA is faster
    // as long as no CTA takes a second tile
    for (int l = 0; l < H.n_levels; ++l) {
        HLevel& L = H.lv[l];
        L.shape = SHAPE_32;
        if (!mg_levels) continue;
        if (l == 0 && H.wide0) {
            L.shape = SHAPE_WIDE;
            continue;
        }
        auto count = [&](int tx, int ty) { return (long long)((L.nx + tx - 1) / tx) * ((L.ny + ty - 1) / ty); };
        if (count(8, 8) <= sms) L.shape = SHAPE_8;
        else if (count(16, 16) <= sms) L.shape = SHAPE_16;
        else if (count(32, 16) <= sms) L.shape = SHAPE_3216;
    }
    // level 0's coefficients persist in shared memory when each wide tile has its own CTA
    const long long wide_tiles = (long long)((nx + TileWide::TX - 1) / TileWide::TX) * ((ny + TileWide::TY - 1) / TileWide::TY);
    H.persist0 = (H.wide0 && wide_tiles <= sms) ? 1 : 0;
    bool aligned = H.n_leaves > 0;
    for (int q = 0; q < H.n_leaves && aligned; ++q)
        aligned = leaves[q] == 128 * q && leaves[q + 1] - leaves[q] == 128;
    H.fused_res = (kind == HK_MULTIGRID && H.wide0 && aligned) ? 1 : 0;
    // the stationary iteration's x and b too, unless a tile overhangs the grid; inside
    // CG every cycle starts from a new right-hand side
    H.keep_x0 = (H.persist0 && kind == HK_MULTIGRID && ny % TileWide::TY == 0) ? 1 : 0;
    H.one_cta = (kind == HK_MULTIGRID && H.coarse_from == 0) ? 1 : 0;
    // CTA 0 holds no level-0 tile when there are more CTAs than tiles: its persistent
    // area then keeps the coarse levels' four coefficient arrays
    H.coarse_persist = (H.persist0 && H.coarse_from > 0 && H.coarse_from < H.n_levels && sms > wide_tiles &&
                        4 * coarse_cells <= 4 * (size_t)TileWide::SN) ? 1 : 0;
    // shared memory: the persistent tile (if any), then the largest of the tree
    // fold, the grid levels' tiles and the coarse levels of CTA 0
    const int n_grid = H.coarse_from < H.n_levels ? H.coarse_from : H.n_levels;
    auto sn_of = [](int shape) {
        switch (shape) {
            case SHAPE_WIDE: return TileWide::SN;
            case SHAPE_3216: return Tile3216::SN;
            case SHAPE_16: return Tile16::SN;
            case SHAPE_8: return Tile8::SN;
            default: return Tile32::SN;
        }
    };
    // the rows of squares that a wide tile's up phase sums sit above the tile's work area
    const size_t rows = (size_t)(kSolveThreads / 32) * kLeafRow;
    // the work area of the grid levels; kept: level-0 arrays that are elsewhere (0, 4 or 6)
    auto tile_work = [&](int kept) {
        size_t w = 0;
        if (!mg_levels) return w;
        for (int l = 0; l < n_grid; ++l)
            w = std::max<size_t>(w, (6 - (l == 0 ? kept : 0)) * (size_t)sn_of(H.lv[l].shape) +
                                        (H.lv[l].shape == SHAPE_WIDE ? rows : 0));
        if (H.coarse_from >= H.n_levels) w = std::max<size_t>(w, 6 * (size_t)Tile32::SN);
        return w;
    };
    auto coarse_work = [&](bool persist) {
        if (!mg_levels || H.coarse_from >= H.n_levels) return (size_t)0;
        return (persist ? 2 : 6) * coarse_cells + (size_t)H.lv[H.coarse_from].n + kFoldScratch +
               (H.one_cta ? (size_t)H.n_slots + H.n_leaves + 2 : 0);
    };
    // in a batched launch a system has fewer CTAs than tiles: no persistent level-0
    // tile (its six arrays are loaded per tile instead)
    smem_batched_ = sizeof(double) * std::max(fold_doubles, std::max(tile_work(0), coarse_work(false)));
    // the tree fold and the V-cycle never run at the same time: one region serves both
    auto solve_smem = [&](int kept) {
        return sizeof(double) * (kept * (size_t)TileWide::SN +
                                 std::max(fold_doubles, std::max(tile_work(kept), coarse_work(kept && H.coarse_persist))));
    };
    int smem_optin = 0;
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    kernel_ = mg_levels ? k_helm_solve<true> : k_helm_solve<false>;
    cudaFuncAttributes fa{};
    cudaFuncGetAttributes(&fa, kernel_);  // static shared memory (the barrier's word) comes first
    // level 0 keeps what fits: everything, its coefficients, or nothing
    auto fits = [&](int kept) { return solve_smem(kept) + fa.sharedSizeBytes <= (size_t)smem_optin; };
    if (H.keep_x0 && !fits(6)) H.keep_x0 = 0;
    if (H.persist0 && !H.keep_x0 && !fits(4)) H.persist0 = H.coarse_persist = 0;
    smem_ = solve_smem(H.keep_x0 ? 6 : (H.persist0 ? 4 : 0));
    if (smem_ + fa.sharedSizeBytes > (size_t)smem_optin) {
        err = "Helmholtz grid too large for the single-pass reduction tree";
        return OC_ERR_UNSUPPORTED;
    }
    if (const cudaError_t e = allow_smem((const void*)kernel_, smem_, dev); e != cudaSuccess) {
        cudaGetLastError();
        err = std::string("Helmholtz solve kernel's shared memory: ") + cudaGetErrorString(e);
        return OC_ERR_CUDA;
    }
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel_, block_, smem_);
    if (per_sm < 1) {
        err = "Helmholtz solve kernel cannot be resident";
        return OC_ERR_CUDA;
    }
    grid_ = mg_levels && H.coarse_from == 0 ? 1 : sms * std::min(per_sm, 2);
    // PCG-Jacobi with the vectors on the chip (its operator relies on a 0/1 mask)
    pcg_ = !refined && kind == HK_PCG_JACOBI && H.unit_mask && !H.big_fold &&
           pcg_plan(leaves, H.n_slots, nx, pcg_plan_);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        err = std::string("Helmholtz init: ") + cudaGetErrorString(e);
        return OC_ERR_CUDA;
    }
    if (refined) {
        refined_ = new RefinedHelm();
        const int rc = refined_->init(nx, ny, dx0, dy0, coef, rtol, max_iter, mask_host, Ku, Kv, err, status);
        if (rc) return rc;
        refined_->set_log(H.log_iters, H.log_conv, H.log_count, H.log_cap);
    }
    return OC_OK;
}

int HelmSolver::grow_log(int cap, cudaStream_t s, std::string& err) {
    if (cap <= hp_.log_cap) return OC_OK;
    int* it = nullptr;
    int* cv = nullptr;
    if (cudaMalloc(&it, sizeof(int) * cap) != cudaSuccess || cudaMalloc(&cv, sizeof(int) * cap) != cudaSuccess) {
        err = "cudaMalloc failed (solve log)";
        return OC_ERR_CUDA;
    }
    cudaMemcpyAsync(it, hp_.log_iters, sizeof(int) * hp_.log_cap, cudaMemcpyDeviceToDevice, s);
    cudaMemcpyAsync(cv, hp_.log_conv, sizeof(int) * hp_.log_cap, cudaMemcpyDeviceToDevice, s);
    cudaStreamSynchronize(s);
    for (auto& p : allocs_) {
        if (p == hp_.log_iters || p == hp_.log_conv) {
            cudaFree(p);
            p = (p == hp_.log_iters) ? (void*)it : (void*)cv;
        }
    }
    bytes_ += sizeof(int) * 2 * (size_t)(cap - hp_.log_cap);
    hp_.log_iters = it;
    hp_.log_conv = cv;
    hp_.log_cap = cap;
    if (refined_) refined_->set_log(hp_.log_iters, hp_.log_conv, hp_.log_count, hp_.log_cap);
    return OC_OK;
}

void HelmSolver::rebuild(cudaStream_t s) {
    if (refined_) {
        refined_->rebuild(s);
        return;
    }
    for (int l = 0; l < hp_.n_levels; ++l) {
        const HLevel& L = hp_.lv[l];
        const HLevel& F = hp_.lv[l > 0 ? l - 1 : 0];
        k_helm_level<<<(L.n + 255) / 256, 256, 0, s>>>(F, L, l > 0 ? 1 : 0, hp_.unit_mask);
    }
}

HelmParams HelmSolver::batched_params(const double* rhs, double* x) const {
    HelmParams H = hp_;
    H.rhs = rhs;
    H.lv[0].x = x;
    H.persist0 = 0;
    H.keep_x0 = 0;
    H.coarse_persist = 0;
    H.warm = warm_ ? 1 : 0;
    return H;
}

int helm_batch_plan(HelmSolver* const* solvers, const double* const* rhs, double* const* x, int n, HelmBatch& b,
                    std::string& err) {
    helm_batch_free(b);
    if (n < 1) {
        err = "a batched solve needs at least one system";
        return OC_ERR_ARG;
    }
    size_t smem = 0;
    double total = 0.0;
    bool mg = false;
    std::vector<HelmParams> hp(n);
    for (int m = 0; m < n; ++m) {
        if (!solvers[m]->batchable()) {
            err = "batched Helmholtz solve: the refined solver has no batched form";
            return OC_ERR_UNSUPPORTED;
        }
        hp[m] = solvers[m]->batched_params(rhs[m], x[m]);
        mg = mg || hp[m].kind == HK_MULTIGRID || hp[m].kind == HK_PCG_MG;
        smem = std::max(smem, solvers[m]->batched_smem());
        total += solvers[m]->work_weight();
    }
    int dev = 0, sms = 0, smem_optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa{};
    const auto kernel = mg ? k_helm_solve_batched<true> : k_helm_solve_batched<false>;
    cudaFuncGetAttributes(&fa, kernel);
    if (smem + fa.sharedSizeBytes > (size_t)smem_optin) {
        err = "batched Helmholtz solve: a system needs more shared memory than a CTA has";
        return OC_ERR_UNSUPPORTED;
    }
    if (const cudaError_t e = allow_smem((const void*)kernel, smem, dev); e != cudaSuccess) {
        cudaGetLastError();
        err = std::string("batched Helmholtz solve kernel's shared memory: ") + cudaGetErrorString(e);
        return OC_ERR_CUDA;
    }
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 512, smem);
    if (per_sm < 1) {
        err = "batched Helmholtz solve kernel cannot be resident";
        return OC_ERR_CUDA;
    }
    const int grid = sms * std::min(per_sm, 2);
    if (n > grid) {
        err = "more systems than co-resident CTAs";
        return OC_ERR_UNSUPPORTED;
    }
    // CTAs in proportion to the cells, at least one each, the remainder to the largest shares
    std::vector<int> share(n, 1);
    int left = grid - n;
    std::vector<double> want(n);
    for (int m = 0; m < n; ++m) want[m] = (grid - n) * solvers[m]->work_weight() / total;
    for (int m = 0; m < n; ++m) {
        const int add = std::min(left, (int)want[m]);
        share[m] += add;
        left -= add;
        want[m] -= add;
    }
    while (left > 0) {
        int best = 0;
        for (int m = 1; m < n; ++m)
            if (want[m] > want[best]) best = m;
        share[best] += 1;
        want[best] -= 1.0;
        --left;
    }
    b.cta_start.assign(n + 1, 0);
    for (int m = 0; m < n; ++m) b.cta_start[m + 1] = b.cta_start[m] + share[m];
    if (cudaMalloc(&b.d_params, sizeof(HelmParams) * n) != cudaSuccess ||
        cudaMalloc(&b.d_cta_start, sizeof(int) * (n + 1)) != cudaSuccess) {
        helm_batch_free(b);
        err = "cudaMalloc failed (batched solve plan)";
        return OC_ERR_CUDA;
    }
    cudaMemcpy(b.d_params, hp.data(), sizeof(HelmParams) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(b.d_cta_start, b.cta_start.data(), sizeof(int) * (n + 1), cudaMemcpyHostToDevice);
    b.n = n;
    b.grid = b.cta_start[n];
    b.smem = smem;
    b.mg = mg;
    return OC_OK;
}

int helm_batch_grid() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return std::max(1, sms);
}

int helm_batch_launch(const HelmBatch& b, cudaStream_t s, std::string& err) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(b.grid);
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = b.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, b.mg ? k_helm_solve_batched<true> : k_helm_solve_batched<false>,
                                             (const HelmParams*)b.d_params, (const int*)b.d_cta_start, b.n);
    if (e != cudaSuccess) {
        err = std::string("batched Helmholtz solve launch: ") + cudaGetErrorString(e);
        return OC_ERR_CUDA;
    }
    return OC_OK;
}

void helm_batch_free(HelmBatch& b) {
    if (b.d_params) cudaFree(b.d_params);
    if (b.d_cta_start) cudaFree(b.d_cta_start);
    b = HelmBatch{};
}

int HelmSolver::solve(const double* rhs, double* x, cudaStream_t s, std::string& err) {
    if (refined_) return refined_->solve(rhs, x, s, err);
    if (pcg_) {
        const HLevel& L = hp_.lv[0];
        PcgParams P{};
        P.nx = L.nx;
        P.ny = L.ny;
        P.n = L.n;
        P.max_iter = hp_.max_iter;
        P.warm = warm_ ? 1 : 0;
        P.coef = hp_.coef;
        P.rtol = hp_.rtol;
        P.dx2 = L.dx2;
        P.dy2 = L.dy2;
        P.mask = L.mask;
        P.Ku = L.Ku;
        P.Kv = L.Kv;
        P.inv_diag = L.inv_diag;
        P.rhs = rhs;
        P.x = x;
        P.r = hp_.r;
        P.z = hp_.z;
        P.Ap = hp_.Ap;
        P.n_leaves = hp_.n_leaves;
        P.n_slots = hp_.n_slots;
        P.leaf_start = hp_.leaf_start;
        P.leaf_slot = hp_.leaf_slot;
        P.leafA = hp_.leafA;
        P.leafB = hp_.leafB;
        P.leafC = hp_.leafC;
        P.own_max = pcg_plan_.own_max;
        P.window = pcg_plan_.window;
        P.leaves_max = pcg_plan_.leaves_max;
        P.lead = pcg_plan_.mode == PCG_ONE ? 0 : L.nx;
        P.bar_count = hp_.bar_count;
        P.status = hp_.status;
        P.wait_cycles = hp_.wait_cycles;
        P.log_iters = hp_.log_iters;
        P.log_conv = hp_.log_conv;
        P.log_count = hp_.log_count;
        P.log_cap = hp_.log_cap;
        const cudaError_t e = pcg_launch(pcg_plan_, P, s);
        if (e != cudaSuccess) {
            err = std::string("Helmholtz PCG launch: ") + cudaGetErrorString(e);
            return OC_ERR_CUDA;
        }
        return OC_OK;
    }
    HelmParams H = hp_;
    H.rhs = rhs;
    H.lv[0].x = x;
    H.warm = warm_ ? 1 : 0;
    // a cooperative launch (every CTA resident, for the grid barriers) through
    // the extensible launch API, which stream capture records into a graph
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid_);
    cfg.blockDim = dim3(block_);
    cfg.dynamicSmemBytes = smem_;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel_, H);
    if (e != cudaSuccess) {
        err = std::string("Helmholtz solve launch: ") + cudaGetErrorString(e);
        return OC_ERR_CUDA;
    }
    return OC_OK;
}

}  // namespace oc
