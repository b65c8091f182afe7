// Device pieces shared by the persistent Helmholtz kernels (helmholtz.cu,
// helm_pcg.cu): the solve's share of a launch, its barrier, the operator at one
// cell and NumPy's pairwise sums.
#pragma once

#include "grid_barrier.cuh"
#include "helmholtz.cuh"

namespace oc {

// ------------------------------------------------------------------ the solve's CTAs
// A solve runs on the CTAs of its launch, or, in a batched launch that solves
// several systems at once, on one system's share of them: s_grid.cta is the
// CTA's index among the solve's CTAs and s_grid.ncta their number. Every
// work-distribution loop and the barrier use these instead of the launch's grid.
struct SolveGrid {
    int cta, ncta;
};
static __shared__ SolveGrid s_grid;

// ------------------------------------------------------------------ level operators
struct Cell {
    int e, ie, iw, jn, js;  // flat index and its four neighbours (periodic)
};

__device__ __forceinline__ Cell cell_of(int nx, int ny, int e) {
    const int j = e / nx, i = e - j * nx;
    Cell c;
    c.e = e;
    c.ie = j * nx + (i + 1 == nx ? 0 : i + 1);
    c.iw = j * nx + (i == 0 ? nx - 1 : i - 1);
    c.jn = (j + 1 == ny ? 0 : j + 1) * nx + i;
    c.js = (j == 0 ? ny - 1 : j - 1) * nx + i;
    return c;
}

__device__ __forceinline__ Cell cell_of(const HLevel& L, int e) { return cell_of(L.nx, L.ny, e); }

// (A x)[e] with x read through L2 (other CTAs write it): VarOperator.apply
// (solvers_var.py:47-53)
__device__ __forceinline__ double apply_at(const HLevel& L, double coef, const double* x, const Cell& c) {
    const double m = L.mask[c.e];
    const double xm = __ldcg(x + c.e) * m;
    const double xe = __ldcg(x + c.ie) * L.mask[c.ie];
    const double xw = __ldcg(x + c.iw) * L.mask[c.iw];
    const double xn = __ldcg(x + c.jn) * L.mask[c.jn];
    const double xs = __ldcg(x + c.js) * L.mask[c.js];
    const double fx = L.Ku[c.e] * (xe - xm);
    const double fxw = L.Ku[c.iw] * (xm - xw);
    const double fy = L.Kv[c.e] * (xn - xm);
    const double fys = L.Kv[c.js] * (xm - xs);
    const double lap = (fx - fxw) / L.dx2 + (fy - fys) / L.dy2;
    return (xm - coef * lap) * m + xm * (1.0 - m);
}

// ------------------------------------------------------------------ pairwise sums
// NumPy's pairwise sums of one leaf (len <= 128 values) of two sets of values
// that the calling warp has staged in shared memory (a and b; b may equal a).
// Lanes 0..7 add set a and lanes 8..15 set b: lane j forms NumPy's interleaved
// accumulator j in its sequential order from consecutive-lane (conflict-free)
// reads, the eight are folded ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)) by shuffles and
// the len mod 8 remaining values added one by one. Lanes 16..31 repeat lanes
// 0..15.
__device__ __forceinline__ double2 leaf_sums(const double* a, const double* b, int len) {
    const int lane = threadIdx.x & 31, j = lane & 7;
    const double* src = (lane & 8) ? b : a;
    double acc = 0.0;
    const int m = len & ~7;
    if (len == 128) {
        double v[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) v[t] = src[8 * t + j];
        acc = v[0];
#pragma unroll
        for (int t = 1; t < 16; ++t) acc = acc + v[t];
    } else if (len >= 8) {
        acc = src[j];
#pragma unroll 4
        for (int t = 8; t < m; t += 8) acc = acc + src[t + j];
    }
    acc = acc + __shfl_xor_sync(0xffffffffu, acc, 1);
    acc = acc + __shfl_xor_sync(0xffffffffu, acc, 2);
    acc = acc + __shfl_xor_sync(0xffffffffu, acc, 4);
    for (int t = m; t < len; ++t) acc = acc + src[t];
    return make_double2(__shfl_sync(0xffffffffu, acc, 0), __shfl_sync(0xffffffffu, acc, 8));
}

// The tree over the leaf sums is NumPy's (split at n/2 rounded down to a multiple
// of 8), embedded in a perfect binary tree of H.n_slots = 2^D slots: a leaf at
// depth d < D takes the first slot of its subtree and the others stay 0, which
// adds nothing (x + 0.0 is x). So one fold serves every grid size: each lane folds
// P consecutive slots in registers, the lanes of a warp fold their subtrees by
// shuffles, and the CTA's warps theirs. Every addition is the tree's left + right.
template <int P>
__device__ __forceinline__ double lane_tree(const double* v) {
    if constexpr (P == 1)
        return v[0];
    else
        return lane_tree<P / 2>(v) + lane_tree<P / 2>(v + P / 2);
}

template <int P>
__device__ __forceinline__ double warp_tree(const double* src, bool global) {
    const int lane = threadIdx.x & 31;
    double v[P];
#pragma unroll
    for (int q = 0; q < P; ++q) v[q] = global ? __ldcg(src + lane * P + q) : src[lane * P + q];
    double x = lane_tree<P>(v);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double y = __shfl_down_sync(0xffffffffu, x, o);
        if ((lane & (2 * o - 1)) == 0) x = x + y;
    }
    return x;  // lane 0 holds the sum
}

// the sums of NSUM leaf buffers (in global memory, read through L2) folded at
// once by a CTA of 16 warps; sm holds 16 * NSUM doubles
template <int P, int NSUM>
__device__ __forceinline__ void slots_fold(int n_slots, const double* const* leaf, double* sm, double* out) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwa = n_slots / (32 * P);  // warps in use: a power of two, at most the CTA's 16
    if (warp < nwa) {
        double x[NSUM];
#pragma unroll
        for (int s = 0; s < NSUM; ++s) x[s] = warp_tree<P>(leaf[s] + warp * 32 * P, true);
        if (lane == 0)
#pragma unroll
            for (int s = 0; s < NSUM; ++s) sm[s * 16 + warp] = x[s];
    }
    __syncthreads();
    // every warp folds the warps' sums itself, so no barrier is needed to hand them out
#pragma unroll
    for (int s = 0; s < NSUM; ++s) {
        double x = (lane & 15) < nwa ? sm[s * 16 + (lane & 15)] : 0.0;
        for (int o = 1; o < nwa; o <<= 1) {
            const double y = __shfl_down_sync(0xffffffffu, x, o);
            if ((lane & (2 * o - 1)) == 0) x = x + y;
        }
        out[s] = __shfl_sync(0xffffffffu, x, 0);
    }
}

template <int NSUM>
__device__ __forceinline__ void slots_fold_any(int n_slots, const double* const* leaf, double* sm, double* out) {
    if (n_slots <= 512) slots_fold<1, NSUM>(n_slots, leaf, sm, out);
    else if (n_slots == 1024) slots_fold<2, NSUM>(n_slots, leaf, sm, out);
    else if (n_slots == 2048) slots_fold<4, NSUM>(n_slots, leaf, sm, out);
    else if (n_slots == 4096) slots_fold<8, NSUM>(n_slots, leaf, sm, out);
    else if (n_slots == 8192) slots_fold<16, NSUM>(n_slots, leaf, sm, out);
    else slots_fold<32, NSUM>(n_slots, leaf, sm, out);
}

}  // namespace oc
