// PCG-Jacobi solve with the vectors kept on the chip (reference
// libs/core/solvers_var.py:181-197; the operator and the stopping test of
// helmholtz.cu, bit-identical to NumPy).
//
// Each CTA owns a contiguous range of NumPy's leaves, so of cells, for the whole
// solve; r and A p (and, when they fit, x and the coefficients) stay in its shared
// memory, and p of the range and of the row above and below it in a window
// there. What bounds an iteration is latency: the two global sums (each a grid
// barrier and a fold) and the chains of one cell's arithmetic. So the
// iteration is arranged around exactly two barriers:
//   1. A p from the window, <p, A p> by leaves          -- barrier, fold: alpha
//   2. x, r, z = r / diag, <r, r> and <r, z> by leaves  -- barrier, folds: beta
//   then p = z + beta p over the window: z of the rows outside the range is read
//   from the owners, and their p is formed again here by the same operations on
//   the same values instead of waiting for a third barrier.
// A warp takes a leaf at a time, its cells and their sum; with every SM at work, where a
// CTA has tens of leaves, the cells are spread over all threads instead, whatever their
// leaf, and the leaves summed afterwards, eight lanes to a leaf. 1000 x 720: 904 us a
// solve by warps, 812 spread; 251 x 187 on a cluster 490 against 560, 128 x 4 on one CTA
// 245 against 309, where the extra barrier and pass cost more than idle warps do.
// (With the vectors in L2, four barriers and two shuffles a value the three took 1326,
// 1023 and 1505 us.)
// The number of CTAs follows the grid size (pcg_plan): one CTA, whose barriers are
// __syncthreads, for the smallest grids; one cluster of up to 16 CTAs, with the
// cluster's hardware barrier; else every SM with the bounded grid barrier.
#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <vector>

#include "helm_common.cuh"
#include "helm_pcg.cuh"

namespace oc {

static constexpr int PCG_THREADS = 512, PCG_WARPS = PCG_THREADS / 32;
static constexpr int LEAF_PAD = 136;  // 128 values, the next buffer in other banks

// one barrier of the solve's CTAs, by the launch's form
template <int MODE>
__device__ __forceinline__ bool pcg_sync(const PcgParams& H) {
    if constexpr (MODE == PCG_ONE) {
        __syncthreads();
        return true;
    } else if constexpr (MODE == PCG_CLUSTER) {
        // hardware barrier of the cluster; release/acquire at cluster scope covers
        // the global memory its CTAs exchange
        asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;\n" ::: "memory");
        return true;
    } else {
        return grid_sync(H.bar_count, H.status, gridDim.x, H.wait_cycles);
    }
}

// the folds of NSUM leaf buffers, the same bits on every thread of the solve
template <int MODE, int NSUM>
__device__ __forceinline__ void pcg_fold(const PcgParams& H, const double* const* leaf, double* sm, double* out) {
    if constexpr (MODE == PCG_ONE) {
        // a single CTA's leaf buffers are in shared memory, at most 128 slots: every warp folds them
#pragma unroll
        for (int s = 0; s < NSUM; ++s) {
            double x;
            if (H.n_slots == 32) x = warp_tree<1>(leaf[s], false);
            else if (H.n_slots == 64) x = warp_tree<2>(leaf[s], false);
            else x = warp_tree<4>(leaf[s], false);
            out[s] = __shfl_sync(0xffffffffu, x, 0);
        }
    } else {
        slots_fold_any<NSUM>(H.n_slots, leaf, sm, out);
    }
}

// NumPy's pairwise sums of the two values f(e) gives per cell, over each of the CTA's
// leaves, into the leaves' slots of outA and outB. Eight lanes sum a leaf, four leaves a
// warp: lane j forms interleaved accumulator j in its sequential order, the eight are
// folded ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)) by shuffles, and the len mod 8 last cells
// are added one by one.
template <class F>
__device__ __forceinline__ void leaf_group_sums(int nlf, const int* lstart, const int* lslot, F f, double* outA,
                                                double* outB) {
    const int lane = threadIdx.x & 31, j = lane & 7;
    for (int l0 = (threadIdx.x >> 5) * 4; l0 < nlf; l0 += PCG_WARPS * 4) {
        const int l = l0 + (lane >> 3);
        const int st = l < nlf ? lstart[l] : 0, len = l < nlf ? lstart[l + 1] - st : 0, m = len & ~7;
        double2 acc = make_double2(0.0, 0.0);
        if (m) {
            acc = f(st + j);
#pragma unroll 5
            for (int t = 8; t < m; t += 8) {
                const double2 v = f(st + t + j);
                acc.x = acc.x + v.x;
                acc.y = acc.y + v.y;
            }
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            acc.x = acc.x + __shfl_xor_sync(0xffffffffu, acc.x, o);
            if (outB) acc.y = acc.y + __shfl_xor_sync(0xffffffffu, acc.y, o);
        }
        for (int t = m; t < len; ++t) {
            const double2 v = f(st + t);
            acc.x = acc.x + v.x;
            acc.y = acc.y + v.y;
        }
        if (j == 0 && l < nlf) {
            outA[lslot[l]] = acc.x;
            if (outB) outB[lslot[l]] = acc.y;
        }
    }
}

// KEEP: PCG_KEEP_ALL x, r, A p and the coefficients in shared memory; PCG_KEEP_RA
// r and A p; PCG_KEEP_P only the window of p
template <int MODE, int KEEP>
__global__ void __launch_bounds__(PCG_THREADS, 1) k_helm_pcg(const PcgParams H) {
    extern __shared__ __align__(16) double s_pcg[];
    const int tid = threadIdx.x;
    const int cta = blockIdx.x, ncta = gridDim.x;
    const int nx = H.nx, n = H.n;
    const int lf0 = (int)((long long)H.n_leaves * cta / ncta), lf1 = (int)((long long)H.n_leaves * (cta + 1) / ncta);
    const int s0 = H.leaf_start[lf0], own = H.leaf_start[lf1] - s0;
    // shared memory: the warps' leaf buffers, fold scratch (or the leaf buffers of
    // a single CTA), the window of p, then what KEEP keeps
    constexpr bool SPREAD = MODE == PCG_GRID;
    const int lane = tid & 31, warp = tid >> 5;
    double* bufs = s_pcg + warp * 2 * LEAF_PAD;
    double* scratch = s_pcg + (SPREAD ? 0 : PCG_WARPS * 2 * LEAF_PAD);
    double* pw = scratch + 3 * 128;
    double* next = pw + H.window;
    double *r, *ap, *x, *ke = nullptr, *kw = nullptr, *kn = nullptr, *ks = nullptr, *id = nullptr;
    if constexpr (KEEP != PCG_KEEP_P) {
        r = next;
        ap = r + H.own_max;
        next = ap + H.own_max;
    } else {
        r = H.r + s0;
        ap = H.Ap + s0;
    }
    if constexpr (KEEP == PCG_KEEP_ALL) {
        x = next;
        ke = x + H.own_max;
        kw = ke + H.own_max;
        kn = kw + H.own_max;
        ks = kn + H.own_max;
        id = ks + H.own_max;
        next = id + H.own_max;
    } else {
        x = H.x + s0;
    }
    // own leaves: where each starts in the range, and its slot
    const int nlf = lf1 - lf0;
    int* lstart = reinterpret_cast<int*>(next);
    int* lslot = lstart + H.leaves_max + 1;
    unsigned char* flag = reinterpret_cast<unsigned char*>(lslot + H.leaves_max + 1);  // 1: wet, 2: last column, 4: first
    for (int t = tid; t <= nlf; t += PCG_THREADS) {
        lstart[t] = H.leaf_start[lf0 + t] - s0;
        if (t < nlf) lslot[t] = H.leaf_slot[lf0 + t];
    }
    double* leafs[3];
    if constexpr (MODE == PCG_ONE) {
        leafs[0] = scratch;
        leafs[1] = scratch + 128;
        leafs[2] = scratch + 256;
        for (int t = tid; t < 3 * 128; t += PCG_THREADS) scratch[t] = 0.0;  // slots without a leaf stay 0
    } else {
        leafs[0] = H.leafA;
        leafs[1] = H.leafB;
        leafs[2] = H.leafC;
    }
    // window position of own cell e, and of the cells north and south of it
    const int lead = MODE == PCG_ONE ? 0 : nx;
    auto north = [&](int w) {
        if constexpr (MODE == PCG_ONE) return w + nx >= n ? w + nx - n : w + nx;
        return w + nx;
    };
    auto south = [&](int w) {
        if constexpr (MODE == PCG_ONE) return w - nx < 0 ? w - nx + n : w - nx;
        return w - nx;
    };
    bool ok = true;
    int iters = 0, conv = 1;
    double rz = 0.0, tol = 0.0;
    if constexpr (MODE == PCG_GRID) grid_sync_begin(H.status);
    for (int e = tid; e < own; e += PCG_THREADS) {
        const int g = s0 + e, i = g % nx;
        const int gw = i == 0 ? g + nx - 1 : g - 1, gs = g - nx < 0 ? g - nx + n : g - nx;
        flag[e] = (unsigned char)((H.mask[g] > 0.0 ? 1 : 0) | (i + 1 == nx ? 2 : 0) | (i == 0 ? 4 : 0));
        if constexpr (KEEP == PCG_KEEP_ALL) {
            ke[e] = H.Ku[g];
            kw[e] = H.Ku[gw];
            kn[e] = H.Kv[g];
            ks[e] = H.Kv[gs];
            id[e] = H.inv_diag[g];
        }
    }
    __syncthreads();
    // b = rhs mask, the residual of the starting iterate (0, or the x given), z = r / diag;
    // |b|^2 and <r, z> by leaves (solvers_var.py:163-168, 181-185)
    for (int e = tid; e < own; e += PCG_THREADS) {
        const int g = s0 + e;
        double re = H.rhs[g] * H.mask[g];
        if (H.warm) {
            HLevel L0;
            L0.mask = H.mask;
            L0.Ku = const_cast<double*>(H.Ku);
            L0.Kv = const_cast<double*>(H.Kv);
            L0.dx2 = H.dx2;
            L0.dy2 = H.dy2;
            re = re - apply_at(L0, H.coef, H.x, cell_of(nx, H.ny, g));
        }
        if constexpr (KEEP == PCG_KEEP_ALL) x[e] = H.warm ? __ldcg(H.x + g) : 0.0;
        const double ze = H.inv_diag[g] * re;
        r[e] = re;
        ap[e] = ze;
        if constexpr (MODE != PCG_ONE) H.z[g] = ze;
    }
    __syncthreads();
    leaf_group_sums(nlf, lstart, lslot, [&](int e) {
        const double b = H.rhs[s0 + e] * H.mask[s0 + e];
        return make_double2(b * b, r[e] * ap[e]);
    }, leafs[0], leafs[1]);
    if constexpr (KEEP != PCG_KEEP_ALL)
        if (!H.warm) {
            __syncthreads();  // x may be the right-hand side's array, which the sums have read
            for (int e = tid; e < own; e += PCG_THREADS) x[e] = 0.0;
        }
    ok = pcg_sync<MODE>(H);
    if (ok) {
        const double* lv[2] = {leafs[0], leafs[1]};
        double f[2];
        pcg_fold<MODE, 2>(H, lv, scratch, f);
        const double norm_b = sqrt(f[0]);
        rz = f[1];
        tol = H.rtol * norm_b;
        if (norm_b != 0.0) conv = 0;
    }
    if (ok && !conv) {
        // p = z over the window
        for (int w = tid; w < H.window_of(own); w += PCG_THREADS) {
            const int e = w - lead;
            int g = s0 + e;
            if (g < 0) g += n;
            if (g >= n) g -= n;
            pw[w] = (e >= 0 && e < own) ? ap[e] : __ldcg(H.z + g);
        }
        for (int it = 1; it <= H.max_iter; ++it) {
            __syncthreads();
            if constexpr (SPREAD) {
                // four of a thread's cells together: all their loads, then the arithmetic and the
                // stores (past the range's end a thread repeats the last cell and stores nothing)
                for (int e0 = tid; e0 < own; e0 += 4 * PCG_THREADS) {
                    double pe[4], de[4], dw[4], dn[4], ds[4], c_e[4], c_w[4], c_n[4], c_s[4], m[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int eq = e0 + q * PCG_THREADS, e = eq < own ? eq : own - 1, w = e + lead;
                        const int fl = flag[e];
                        m[q] = (fl & 1) ? 1.0 : 0.0;
                        if constexpr (KEEP == PCG_KEEP_ALL) {
                            c_e[q] = ke[e];
                            c_w[q] = kw[e];
                            c_n[q] = kn[e];
                            c_s[q] = ks[e];
                        } else {
                            const int g = s0 + e;
                            c_e[q] = __ldg(H.Ku + g);
                            c_w[q] = __ldg(H.Ku + ((fl & 4) ? g + nx - 1 : g - 1));
                            c_n[q] = __ldg(H.Kv + g);
                            c_s[q] = __ldg(H.Kv + (g - nx < 0 ? g - nx + n : g - nx));
                        }
                        pe[q] = pw[w];
                        de[q] = pw[(fl & 2) ? w + 1 - nx : w + 1];
                        dw[q] = pw[(fl & 4) ? w - 1 + nx : w - 1];
                        dn[q] = pw[north(w)];
                        ds[q] = pw[south(w)];
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int e = e0 + q * PCG_THREADS;
                        if (e >= own) break;
                        // VarOperator.apply (solvers_var.py:47-53); p is 0 on dry cells
                        // (z = r / diag, and r is a masked difference), so p mask is p
                        const double fx = c_e[q] * (de[q] - pe[q]);
                        const double fxw = c_w[q] * (pe[q] - dw[q]);
                        const double fy = c_n[q] * (dn[q] - pe[q]);
                        const double fys = c_s[q] * (pe[q] - ds[q]);
                        const double lap = (fx - fxw) / H.dx2 + (fy - fys) / H.dy2;
                        ap[e] = (pe[q] - H.coef * lap) * m[q] + pe[q] * (1.0 - m[q]);
                    }
                }
                __syncthreads();
                leaf_group_sums(nlf, lstart, lslot, [&](int e) { return make_double2(pw[e + lead] * ap[e], 0.0); }, leafs[2],
                                nullptr);
            } else {
                for (int L = warp; L < nlf; L += PCG_WARPS) {
                    const int st = lstart[L], len = lstart[L + 1] - st;
                    // a lane's four cells together: all their loads, then the arithmetic, then
                    // the stores (past the leaf's end a lane repeats its last cell and stores nothing)
                    double pe[4], de[4], dw[4], dn[4], ds[4], c_e[4], c_w[4], c_n[4], c_s[4], m[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int t = lane + 32 * q, e = st + (t < len ? t : len - 1), w = e + lead;
                        const int fl = flag[e];
                        m[q] = (fl & 1) ? 1.0 : 0.0;
                        if constexpr (KEEP == PCG_KEEP_ALL) {
                            c_e[q] = ke[e];
                            c_w[q] = kw[e];
                            c_n[q] = kn[e];
                            c_s[q] = ks[e];
                        } else {
                            const int g = s0 + e;
                            c_e[q] = __ldg(H.Ku + g);
                            c_w[q] = __ldg(H.Ku + ((fl & 4) ? g + nx - 1 : g - 1));
                            c_n[q] = __ldg(H.Kv + g);
                            c_s[q] = __ldg(H.Kv + (g - nx < 0 ? g - nx + n : g - nx));
                        }
                        pe[q] = pw[w];
                        de[q] = pw[(fl & 2) ? w + 1 - nx : w + 1];
                        dw[q] = pw[(fl & 4) ? w - 1 + nx : w - 1];
                        dn[q] = pw[north(w)];
                        ds[q] = pw[south(w)];
                    }
                    double av[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        // VarOperator.apply (solvers_var.py:47-53); p is 0 on dry cells
                        // (z = r / diag, and r is a masked difference), so p mask is p
                        const double fx = c_e[q] * (de[q] - pe[q]);
                        const double fxw = c_w[q] * (pe[q] - dw[q]);
                        const double fy = c_n[q] * (dn[q] - pe[q]);
                        const double fys = c_s[q] * (pe[q] - ds[q]);
                        const double lap = (fx - fxw) / H.dx2 + (fy - fys) / H.dy2;
                        av[q] = (pe[q] - H.coef * lap) * m[q] + pe[q] * (1.0 - m[q]);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int t = lane + 32 * q;
                        if (t < len) {
                            ap[st + t] = av[q];
                            bufs[t] = pe[q] * av[q];
                        }
                    }
                    __syncwarp();
                    const double2 sums = leaf_sums(bufs, bufs, len);
                    if (lane == 0) leafs[2][lslot[L]] = sums.x;
                    __syncwarp();
                }
            }
            ok = pcg_sync<MODE>(H);
            if (!ok) break;
            double pap[1];
            {
                const double* lv[1] = {leafs[2]};
                pcg_fold<MODE, 1>(H, lv, scratch, pap);
            }
            const double alpha = rz / pap[0];
            if constexpr (SPREAD) {
                for (int e0 = tid; e0 < own; e0 += 4 * PCG_THREADS) {
                    double xe[4], re[4], pe[4], ae[4], di[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int eq = e0 + q * PCG_THREADS, e = eq < own ? eq : own - 1;
                        xe[q] = x[e];
                        re[q] = r[e];
                        pe[q] = pw[e + lead];
                        ae[q] = ap[e];
                        if constexpr (KEEP == PCG_KEEP_ALL) di[q] = id[e];
                        else di[q] = __ldg(H.inv_diag + s0 + e);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int e = e0 + q * PCG_THREADS;
                        if (e >= own) break;
                        const double rn = re[q] - alpha * ae[q];
                        const double ze = di[q] * rn;
                        x[e] = xe[q] + alpha * pe[q];
                        r[e] = rn;
                        ap[e] = ze;  // z, until the next A p
                        // the rows a neighbouring range reads
                        if constexpr (MODE != PCG_ONE)
                            if (e < nx || e >= own - nx) H.z[s0 + e] = ze;
                    }
                }
                __syncthreads();
                leaf_group_sums(nlf, lstart, lslot, [&](int e) {
                    const double re = r[e];
                    return make_double2(re * re, re * ap[e]);
                }, leafs[0], leafs[1]);
            } else {
                for (int L = warp; L < nlf; L += PCG_WARPS) {
                    const int st = lstart[L], len = lstart[L + 1] - st;
                    double xe[4], re[4], pe[4], ae[4], di[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int t = lane + 32 * q, e = st + (t < len ? t : len - 1);
                        xe[q] = x[e];
                        re[q] = r[e];
                        pe[q] = pw[e + lead];
                        ae[q] = ap[e];
                        if constexpr (KEEP == PCG_KEEP_ALL) di[q] = id[e];
                        else di[q] = __ldg(H.inv_diag + s0 + e);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int t = lane + 32 * q;
                        if (t < len) {
                            const int e = st + t;
                            const double rn = re[q] - alpha * ae[q];
                            const double ze = di[q] * rn;
                            x[e] = xe[q] + alpha * pe[q];
                            r[e] = rn;
                            ap[e] = ze;  // z, until the next A p
                            // the rows a neighbouring range reads
                            if constexpr (MODE != PCG_ONE)
                                if (e < nx || e >= own - nx) H.z[s0 + e] = ze;
                            bufs[t] = rn * rn;
                            bufs[LEAF_PAD + t] = rn * ze;
                        }
                    }
                    __syncwarp();
                    const double2 sums = leaf_sums(bufs, bufs + LEAF_PAD, len);
                    if (lane == 0) {
                        leafs[0][lslot[L]] = sums.x;
                        leafs[1][lslot[L]] = sums.y;
                    }
                    __syncwarp();
                }
            }
            ok = pcg_sync<MODE>(H);
            if (!ok) break;
            iters = it;
            double f[2];
            {
                const double* lv[2] = {leafs[0], leafs[1]};
                pcg_fold<MODE, 2>(H, lv, scratch, f);
            }
            if (sqrt(f[0]) <= tol) {
                conv = 1;
                break;
            }
            const double beta = f[1] / rz;
            rz = f[1];
            // the rows outside the range first: their z is on its way while the range's own is used
            if constexpr (MODE != PCG_ONE) {
                constexpr int K = 4;
                for (int h0 = tid; h0 < 2 * nx; h0 += K * PCG_THREADS) {
                    double z[K];
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const int h = h0 + k * PCG_THREADS;
                        int g = h < nx ? s0 - nx + h : s0 + own + h - nx;
                        if (g < 0) g += n;
                        if (g >= n) g -= n;
                        z[k] = h < 2 * nx ? __ldcg(H.z + g) : 0.0;
                    }
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        const int h = h0 + k * PCG_THREADS, w = h < nx ? h : own + h;
                        if (h < 2 * nx) pw[w] = z[k] + beta * pw[w];
                    }
                }
            }
#pragma unroll 4
            for (int e = tid; e < own; e += PCG_THREADS) pw[e + lead] = ap[e] + beta * pw[e + lead];
        }
    }
    if constexpr (KEEP == PCG_KEEP_ALL) {
        __syncthreads();
        for (int e = tid; e < own; e += PCG_THREADS) H.x[s0 + e] = x[e];
    }
    if constexpr (MODE == PCG_GRID) grid_sync_end(H.bar_count, cta == 0);
    if (cta == 0 && tid == 0) {
        const int idx = *H.log_count;
        if (idx < H.log_cap) {
            H.log_iters[idx] = ok ? iters : -1;
            H.log_conv[idx] = ok ? conv : 0;
        }
        *H.log_count = idx + 1;
    }
    // no CTA of a cluster leaves while another may still wait for its arrival: the
    // last barrier was passed by all before any left the loop
}

// ------------------------------------------------------------------ host side
typedef void (*PcgKernel)(const PcgParams);

static PcgKernel pcg_kernel(int mode, int keep) {
    if (mode == PCG_ONE) return k_helm_pcg<PCG_ONE, PCG_KEEP_ALL>;
    if (mode == PCG_CLUSTER) return k_helm_pcg<PCG_CLUSTER, PCG_KEEP_ALL>;
    return keep == PCG_KEEP_ALL  ? (PcgKernel)k_helm_pcg<PCG_GRID, PCG_KEEP_ALL>
           : keep == PCG_KEEP_RA ? (PcgKernel)k_helm_pcg<PCG_GRID, PCG_KEEP_RA>
                                 : (PcgKernel)k_helm_pcg<PCG_GRID, PCG_KEEP_P>;
}

// shared memory of a launch whose largest range has `own` cells, window `window` and `leaves` leaves
static size_t pcg_smem(int mode, int keep, size_t own, size_t window, size_t leaves) {
    const size_t doubles = (mode == PCG_GRID ? 0 : PCG_WARPS * 2 * LEAF_PAD) + 3 * 128 + window +
                           (keep == PCG_KEEP_ALL ? 8 * own : (keep == PCG_KEEP_RA ? 2 * own : 0));
    return doubles * sizeof(double) + 2 * (leaves + 1) * sizeof(int) + ((own + 15) & ~(size_t)15);
}

// the kernels' shared-memory allowance on this device; it only grows, so every
// solver's launches stay valid
static bool pcg_allow(PcgKernel k, size_t smem, int dev) {
    static std::mutex mu;
    static std::map<std::pair<int, PcgKernel>, size_t> allowance;
    std::lock_guard<std::mutex> lock(mu);
    size_t& a = allowance[{dev, k}];
    if (smem > a) {
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
            cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        a = smem;
    }
    return true;
}

static bool pcg_try(int mode, int keep, int ncta, const std::vector<int>& leaves, int nx, int dev, size_t optin,
                    PcgPlan& plan) {
    const int n_leaves = (int)leaves.size() - 1;
    if (ncta > n_leaves) return false;
    int own = 0, most = 0;
    for (int c = 0; c < ncta; ++c) {
        const int a = (int)((long long)n_leaves * c / ncta), b = (int)((long long)n_leaves * (c + 1) / ncta);
        own = std::max(own, leaves[b] - leaves[a]);
        most = std::max(most, b - a);
    }
    const int n = leaves.back();
    const int window = mode == PCG_ONE ? n : own + 2 * nx;
    // a window must not meet itself: its rows above and below belong to other ranges
    if (mode != PCG_ONE && window > n) return false;
    const size_t smem = pcg_smem(mode, keep, (size_t)own, (size_t)window, (size_t)most);
    cudaFuncAttributes fa{};
    PcgKernel k = pcg_kernel(mode, keep);
    if (cudaFuncGetAttributes(&fa, k) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    if (smem + fa.sharedSizeBytes > optin || !pcg_allow(k, smem, dev)) return false;
    plan = PcgPlan{mode, keep, ncta, own, window, most, smem};
    return true;
}

bool pcg_plan(const std::vector<int>& leaves, int n_slots, int nx, PcgPlan& plan) {
    const int n = leaves.back();
    int dev = 0, sms = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (n <= PCG_ONE_CELLS && n_slots <= 128 && pcg_try(PCG_ONE, PCG_KEEP_ALL, 1, leaves, nx, dev, (size_t)optin, plan))
        return true;
    if (n <= PCG_CLUSTER_CELLS) {
        for (int c : {16, 8}) {
            if (!pcg_try(PCG_CLUSTER, PCG_KEEP_ALL, c, leaves, nx, dev, (size_t)optin, plan)) continue;
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(c);
            cfg.blockDim = dim3(PCG_THREADS);
            cfg.dynamicSmemBytes = plan.smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = (unsigned)c;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            int clusters = 0;
            if (cudaOccupancyMaxActiveClusters(&clusters, (const void*)pcg_kernel(PCG_CLUSTER, PCG_KEEP_ALL), &cfg) ==
                    cudaSuccess && clusters >= 1)
                return true;
            cudaGetLastError();
        }
    }
    for (int keep : {PCG_KEEP_ALL, PCG_KEEP_RA, PCG_KEEP_P})
        if (pcg_try(PCG_GRID, keep, std::min(sms, (int)leaves.size() - 1), leaves, nx, dev, (size_t)optin, plan)) {
            int per_sm = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pcg_kernel(PCG_GRID, keep), PCG_THREADS, plan.smem);
            if (per_sm >= 1) return true;
        }
    return false;
}

cudaError_t pcg_launch(const PcgPlan& plan, const PcgParams& H, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(plan.ncta);
    cfg.blockDim = dim3(PCG_THREADS);
    cfg.dynamicSmemBytes = plan.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    if (plan.mode == PCG_GRID) {
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
    } else {
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = (unsigned)plan.ncta;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, pcg_kernel(plan.mode, plan.keep), H);
}

}  // namespace oc
