// The V(2,2) cycle of the Helmholtz solve (reference libs/core/solvers_var.py:
// 118-152), device side; helmholtz.cu includes it.
//
// A fine level is processed tile by tile in shared memory. The down phase loads x,
// b and the coefficients of a tile plus a HALO-wide ring, runs the two
// pre-smoothing sweeps (four red-black half-sweeps) on a region that shrinks by one
// cell per half-sweep, and forms the restricted residual of the interior; the up
// phase adds the prolonged coarse correction and runs the two reverse
// post-smoothing sweeps the same way. Every value in the valid region is the one
// the whole-grid sweep produces (same inputs, same operations), so the result is
// that of sweeping the level with a grid barrier between half-sweeps, with two
// barriers per level instead of nine. Levels of at most kCoarseCells cells run
// inside CTA 0; a stationary solve of at most kOneCtaCells cells runs wholly in one CTA.
//
// A half-sweep is bound by shared-memory bandwidth (ten reads and a write per
// updated cell), so the two colours of every array are stored apart: cell (i, j) of
// colour p = (i + j) mod 2 at [p][j][i / 2]. A half-sweep then reads and writes
// consecutive words where the natural order strides by two (twice the passes
// through the banks), and a cell's neighbours are all of the other colour, at the
// same position up to one. A level with an odd size has no such order (the wrap
// changes colours); only a coarsest level can be odd, and it keeps the flat order.
//
// What a cycle spends its time on is latency: a grid barrier is about 3000 cycles, a
// half-sweep of one cell per thread 500, a tile's loads 1000 to 1500. Hence the fewest
// barriers and loads: the residual's test runs beside the next cycle's first phase, a
// wide level-0 tile keeps its x and b in shared memory, CTA 0 keeps the coarse levels'
// coefficients wherever it has no tile, and what a phase needs of a level's geometry
// stands in a table. us a solve (V-cycles), before and with these: 48 x 48 (50) 1199 and
// 932, 128 x 128 (12) 562 and 427, 256 x 256 727 and 586, 512 x 512 (12) 934 and 837.
#pragma once

#include "helm_common.cuh"

namespace oc {

// The phases below are calls (inlined together they would spill), so they name the
// solve's shared memory themselves: a pointer passed in would be a generic one. Areas
// of it are offsets in doubles, -1 for none; the solve's parameters are s_helm.
extern __shared__ double smem_all[];
static __shared__ HelmParams s_helm;

static constexpr int kCoarseCells = 1024;
// fine-level tiles: interior TX x TY cells plus a halo of HALO cells, enough
// for four red-black half-sweeps and one residual on a shrinking region
static constexpr int HALO = 5;
template <int TX_, int TY_>
struct TileShape {
    static constexpr int TX = TX_, TY = TY_;
    static constexpr int RW = TX + 2 * HALO, RH = TY + 2 * HALO, RN = RW * RH;
    // one colour: HW cells per row, CN values, 8 mod 16 so that the halves of a warp
    // that reads both colours of a row meet different banks
    static constexpr int HW = RW / 2;
    static constexpr int CN = ((HW * RH + 7) / 16) * 16 + 8;
    static constexpr int SN = 2 * CN;
    static_assert(CN >= HW * RH && RW % 2 == 0 && TX % 2 == 0 && TY % 2 == 0, "colour layout");
    // position of region cell (ri, rj); tiles start at even cells of even-sized levels,
    // so the colour follows from the region coordinates
    static __device__ __forceinline__ int pos(int ri, int rj) { return ((ri + rj) & 1) * CN + rj * HW + (ri >> 1); }
};
using Tile32 = TileShape<32, 32>;
using Tile3216 = TileShape<32, 16>;
using Tile16 = TileShape<16, 16>;
using Tile8 = TileShape<8, 8>;
using TileWide = TileShape<128, 16>;  // level 0 of large grids: one tile per CTA, one NumPy leaf per row
// per-level tile shape codes (HLevel::shape)
enum { SHAPE_32 = 0, SHAPE_3216 = 1, SHAPE_16 = 2, SHAPE_8 = 3, SHAPE_WIDE = 4 };

// ------------------------------------------------------------------ asynchronous copies
// cp.async into shared memory without a register round trip, so a thread's
// copies are all in flight at once. The 8-byte form goes through L1, which is not
// coherent with other SMs' writes, so it serves only arrays that stay constant
// during the solve (the level coefficients); b and x, which other CTAs of the
// launch write, are read through L2 (__ldcg).
__device__ __forceinline__ void cpa_ca8(double* sdst, const double* gsrc) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cpa_wait_all() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}

__device__ __forceinline__ int wrap_any(int i, int n) {
    if (i >= 0 && i < n) return i;
    if (i < 0 && i + n >= 0) return i + n;
    if (i >= n && i - n < n) return i - n;
    const int r = i % n;
    return r < 0 ? r + n : r;
}

// a tile's (or a coarse level's) arrays; id is 1 / diagonal times the mask
// (HLevel::idm), which makes the mask multiply of a half-sweep part of it
struct TileRefs {
    double *x, *b, *ku, *kv, *id, *m;
};

// the coefficients from `coef` on, x and b from `xb` on
__device__ __forceinline__ TileRefs tile_refs(int coef, int xb, int stride) {
    double *cb = smem_all + coef, *base = smem_all + xb;
    TileRefs t;
    t.ku = cb;
    t.kv = cb + stride;
    t.id = cb + 2 * stride;
    t.m = cb + 3 * stride;
    t.x = base;
    t.b = base + stride;
    return t;
}

// the arrays of a tile: all of them in the work area, or, of a persistent tile, the
// coefficients (and with H.keep_x0 x and b) in its persistent area
template <class S>
__device__ __forceinline__ TileRefs tile_arrays(int smem, int persist) {
    if (persist < 0) return tile_refs(smem, smem + 4 * S::SN, S::SN);
    return tile_refs(persist, s_helm.keep_x0 ? persist + 4 * S::SN : smem, S::SN);
}

// ------------------------------------------------------------------ tiles, colours apart
// The tile region of level L whose interior starts at (i0, j0): x from xin (or zero),
// plus the coarse correction e * mask when the coarse level's x (xc, rows of cnx) is
// given; the coefficients by
// asynchronous copies unless they are in place already (COEF false). All of a
// thread's loads are issued before its first store to shared memory.
template <class S, bool COEF>
__device__ __forceinline__ void tile_load(const HLevel& L, int i0, int j0, const double* xin, const double* xc,
                                          int cnx, TileRefs t) {
    constexpr int K = (S::RN + kSolveThreads - 1) / kSolveThreads;
    double xv[K], bv[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int r = threadIdx.x + k * kSolveThreads;
        xv[k] = bv[k] = 0.0;
        if (r >= S::RN) continue;
        const int rj = r / S::RW, ri = r - rj * S::RW;
        const int gi = wrap_any(i0 - HALO + ri, L.nx), gj = wrap_any(j0 - HALO + rj, L.ny);
        const int g = gj * L.nx + gi, o = S::pos(ri, rj);
        if (COEF) {
            cpa_ca8(t.ku + o, L.Ku + g);
            cpa_ca8(t.kv + o, L.Kv + g);
            cpa_ca8(t.id + o, L.idm + g);
            cpa_ca8(t.m + o, L.mask + g);
        }
        double x = xin ? __ldcg(xin + g) : 0.0;
        if (xc) x = x + __ldcg(xc + (gj >> 1) * cnx + (gi >> 1)) * __ldg(L.mask + g);
        xv[k] = x;
        bv[k] = __ldcg(L.b + g);
    }
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int r = threadIdx.x + k * kSolveThreads;
        if (r >= S::RN) continue;
        const int rj = r / S::RW, ri = r - rj * S::RW;
        const int o = S::pos(ri, rj);
        t.x[o] = xv[k];
        t.b[o] = bv[k];
    }
    if (COEF) cpa_wait_all();
    __syncthreads();
}

// The phases of a level-0 tile whose x and b stay in its CTA's shared memory for the
// solve (H.keep_x0): only the ring's x is read again, and the coarse correction.
template <class S>
__device__ __forceinline__ void tile_refresh(const HLevel& L, int i0, int j0, const double* xin, const double* xc,
                                             int cnx, TileRefs t) {
    constexpr int NR = S::RN - S::TX * S::TY, KR = (NR + kSolveThreads - 1) / kSolveThreads;
    constexpr int KI = (S::TX * S::TY + kSolveThreads - 1) / kSolveThreads;
    constexpr int BAND = 2 * HALO * S::RW;  // the rows above and below the interior, then the columns beside it
    auto ring = [&](int h, int& ri, int& rj) {
        if (h < BAND) {
            rj = h / S::RW;
            ri = h - rj * S::RW;
            if (rj >= HALO) rj += S::TY;
        } else {
            h -= BAND;
            rj = h / (2 * HALO);
            ri = h - rj * (2 * HALO);
            rj += HALO;
            if (ri >= HALO) ri += S::TX;
        }
    };
    double xv[KR], cv[KI];
#pragma unroll
    for (int k = 0; k < KR; ++k) {
        const int h = threadIdx.x + k * kSolveThreads;
        xv[k] = 0.0;
        if (h >= NR) continue;
        int ri, rj;
        ring(h, ri, rj);
        const int gi = wrap_any(i0 - HALO + ri, L.nx), gj = wrap_any(j0 - HALO + rj, L.ny);
        xv[k] = __ldcg(xin + gj * L.nx + gi);
        if (xc) xv[k] = xv[k] + __ldcg(xc + (gj >> 1) * cnx + (gi >> 1)) * t.m[S::pos(ri, rj)];
    }
    if (xc) {
#pragma unroll
        for (int k = 0; k < KI; ++k) {
            const int h = threadIdx.x + k * kSolveThreads;
            if (h >= S::TX * S::TY) continue;
            const int cj = h / S::TX, ci = h - cj * S::TX;
            cv[k] = __ldcg(xc + ((j0 + cj) >> 1) * cnx + ((i0 + ci) >> 1));
        }
    }
#pragma unroll
    for (int k = 0; k < KR; ++k) {
        const int h = threadIdx.x + k * kSolveThreads;
        if (h >= NR) continue;
        int ri, rj;
        ring(h, ri, rj);
        t.x[S::pos(ri, rj)] = xv[k];
    }
    if (xc) {
#pragma unroll
        for (int k = 0; k < KI; ++k) {
            const int h = threadIdx.x + k * kSolveThreads;
            if (h >= S::TX * S::TY) continue;
            const int cj = h / S::TX, ci = h - cj * S::TX;
            const int o = S::pos(ci + HALO, cj + HALO);
            t.x[o] = t.x[o] + cv[k] * t.m[o];
        }
    }
    __syncthreads();
}

// one red-black half-sweep of colour p on the rows of ring >= SHRINK. Cells of the
// outer columns are updated too; their values are invalid, as are all values of
// rings < SHRINK, and no valid cell reads them again.
template <class S, int SHRINK>
__device__ __forceinline__ void tile_half_sweep(const HLevel& L, TileRefs t, int p, bool unit) {
    constexpr int HW = S::HW, CN = S::CN;
    double* xp = t.x + p * CN;
    const double* xo = t.x + (1 - p) * CN;
    const double *kup = t.ku + p * CN, *kuo = t.ku + (1 - p) * CN;
    const double *kvp = t.kv + p * CN, *kvo = t.kv + (1 - p) * CN;
    const double *bp = t.b + p * CN, *ip = t.id + p * CN;
    const double cx = L.cx, cy = L.cy;
    constexpr int N = (S::RH - 2 * SHRINK) * HW, K = (N + kSolveThreads - 1) / kSolveThreads;
    double v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int r = threadIdx.x + k * kSolveThreads;
        v[k] = 0.0;
        if (r < N) {
            const int q = SHRINK * HW + r;
            const int e = q + ((p + q / HW) & 1);  // the east neighbour; the west one sits before it
            const double nb = cx * (kup[q] * xo[e] + kuo[e - 1] * xo[e - 1]) +
                              cy * (kvp[q] * xo[q + HW] + kvo[q - HW] * xo[q - HW]);
            v[k] = ip[q] * (bp[q] + nb);
            if (!unit) v[k] = v[k] * t.m[p * CN + q];
        }
    }
    // stored only now: a store would hold back the next cell's loads
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const int r = threadIdx.x + k * kSolveThreads;
        if (r < N) xp[SHRINK * HW + r] = v[k];
    }
    __syncthreads();
}

// four half-sweeps with colours c0, 1 - c0, c0, 1 - c0 on a region shrinking by one ring each
template <class S>
__device__ __forceinline__ void tile_four_half_sweeps(const HLevel& L, TileRefs t, int c0, bool unit) {
    tile_half_sweep<S, 1>(L, t, c0, unit);
    tile_half_sweep<S, 2>(L, t, 1 - c0, unit);
    tile_half_sweep<S, 3>(L, t, c0, unit);
    tile_half_sweep<S, 4>(L, t, 1 - c0, unit);
}

// (b - A x) * mask (VarOperator.apply, solvers_var.py:47-53) from a cell's own values
// and its neighbours'. The caller's x carries the mask already when masks are 0/1
// (every half-sweep ends with it).
__device__ __forceinline__ double residual_of(const HLevel& L, double coef, double m, double b, double xm, double xe,
                                              double xw, double xn, double xs, double ke, double kw, double kn,
                                              double ks) {
    const double fx = ke * (xe - xm);
    const double fxw = kw * (xm - xw);
    const double fy = kn * (xn - xm);
    const double fys = ks * (xm - xs);
    const double lap = (fx - fxw) / L.dx2 + (fy - fys) / L.dy2;
    const double ax = (xm - coef * lap) * m + xm * (1.0 - m);
    return (b - ax) * m;
}

// at region cell (ri, rj) of the interior
template <class S>
__device__ __forceinline__ double tile_residual(const HLevel& L, double coef, TileRefs t, int ri, int rj, bool unit) {
    constexpr int HW = S::HW, CN = S::CN;
    const int p = (ri + rj) & 1, q = rj * HW + (ri >> 1), e = q + (ri & 1);
    const int op = p * CN, oo = (1 - p) * CN;
    const double* x = t.x;
    const double m = t.m[op + q];
    double xm = x[op + q], xe = x[oo + e], xw = x[oo + e - 1], xn = x[oo + q + HW], xs = x[oo + q - HW];
    if (!unit) {
        xm = xm * m;
        xe = xe * t.m[oo + e];
        xw = xw * t.m[oo + e - 1];
        xn = xn * t.m[oo + q + HW];
        xs = xs * t.m[oo + q - HW];
    }
    return residual_of(L, coef, m, t.b[op + q], xm, xe, xw, xn, xs, t.ku[op + q], t.ku[oo + e - 1], t.kv[op + q],
                       t.kv[oo + q - HW]);
}

template <class S>
__device__ __forceinline__ void tile_store_x(const HLevel& L, int i0, int j0, TileRefs t, double* xout) {
    for (int r = threadIdx.x; r < S::TX * S::TY; r += kSolveThreads) {
        const int cj = r / S::TX, ci = r - cj * S::TX;
        const int gi = i0 + ci, gj = j0 + cj;
        if (gi >= L.nx || gj >= L.ny) continue;
        xout[gj * L.nx + gi] = t.x[S::pos(ci + HALO, cj + HALO)];
    }
}

// With a CTA of its own for every level-0 tile, the tiles go to the last CTAs
// (tile = CTA - (CTAs - tiles)), so CTA 0, which runs the coarse levels, keeps
// its persistent region for their coefficients (H.coarse_persist).
__device__ __forceinline__ int level0_tile_of_cta(int tiles) { return s_grid.cta - (s_grid.ncta - tiles); }

// The first tile of this CTA. With a CTA to spare the tiles go to the last CTAs: the first
// ones form the residual sums meanwhile, and CTA 0 keeps its shared memory to itself.
__device__ __forceinline__ int first_tile(int tiles) {
    return tiles < s_grid.ncta ? s_grid.ncta - 1 - s_grid.cta : s_grid.cta;
}

__device__ __forceinline__ int level_tiles(const HLevel& L) {
    int tx = 32, ty = 32;
    if (L.shape == SHAPE_WIDE) tx = TileWide::TX, ty = TileWide::TY;
    else if (L.shape == SHAPE_3216) ty = 16;
    else if (L.shape == SHAPE_16) tx = ty = 16;
    else if (L.shape == SHAPE_8) tx = ty = 8;
    return ((L.nx + tx - 1) / tx) * ((L.ny + ty - 1) / ty);
}

// Level 0's coefficients (and, with H.keep_x0, its x and b) stay in shared memory for
// a whole solve when every level-0 tile has a CTA of its own (H.persist0).
__device__ __noinline__ void persist_level0(int smem, int persist) {
    using S = TileWide;
    const HelmParams& H = s_helm;
    const HLevel& L = H.lv[0];
    const int tx = (L.nx + S::TX - 1) / S::TX;
    const int tile = level0_tile_of_cta(tx * ((L.ny + S::TY - 1) / S::TY));
    if (tile < 0) return;
    tile_load<S, true>(L, (tile % tx) * S::TX, (tile / tx) * S::TY, L.x, nullptr, 0, tile_arrays<S>(smem, persist));
}

// down phase of level l: pre-smoothing, restricted residual into level l+1
// (solvers_var.py:141-147); x of level l+1 starts at zero implicitly
template <class S>
__device__ __noinline__ void mg_down(int l, const double* xin, double* xout, int smem, int persist) {
    const HelmParams& H = s_helm;
    const HLevel& L = H.lv[l];
    const HLevel& C = H.lv[l + 1];
    const bool unit = H.unit_mask != 0;
    const int tx = (L.nx + S::TX - 1) / S::TX, ty = (L.ny + S::TY - 1) / S::TY;
    const bool keep = persist >= 0;
    const TileRefs t = tile_arrays<S>(smem, persist);
    for (int tile = keep ? level0_tile_of_cta(tx * ty) : first_tile(tx * ty); tile < tx * ty; tile += s_grid.ncta) {
        if (tile < 0) continue;  // CTA-uniform: this CTA holds no persistent tile
        const int i0 = (tile % tx) * S::TX, j0 = (tile / tx) * S::TY;
        if (!keep) tile_load<S, true>(L, i0, j0, xin, nullptr, 0, t);
        else if constexpr (S::TX == TileWide::TX) {
            if (H.keep_x0) tile_refresh<S>(L, i0, j0, xin, nullptr, 0, t);
            else tile_load<S, false>(L, i0, j0, xin, nullptr, 0, t);
        }
        tile_four_half_sweeps<S>(L, t, 0, unit);
        tile_store_x<S>(L, i0, j0, t, xout);
        constexpr int NC = (S::TX / 2) * (S::TY / 2);  // coarse cells of the tile
        if constexpr (4 * NC <= 1024 && (4 * NC) % 32 == 0 && S::TX != TileWide::TX) {
            // four lanes per coarse cell, one child residual each, summed by the
            // first of them in the order a + b + c + d (the loop bound is a
            // multiple of 32, so whole warps take part in the shuffles)
            for (int q = threadIdx.x; q < 4 * NC; q += kSolveThreads) {
                const int r = q >> 2, child = q & 3;
                const int cj = r / (S::TX / 2), ci = r - cj * (S::TX / 2);
                const int I = i0 / 2 + ci, J = j0 / 2 + cj;
                const double val = tile_residual<S>(L, H.coef, t, HALO + 2 * ci + (child & 1),
                                                    HALO + 2 * cj + (child >> 1), unit);
                const double b = __shfl_down_sync(0xffffffffu, val, 1);
                const double c = __shfl_down_sync(0xffffffffu, val, 2);
                const double d = __shfl_down_sync(0xffffffffu, val, 3);
                if (child == 0 && I < C.nx && J < C.ny) C.b[J * C.nx + I] = 0.25 * (val + b + c + d);
            }
        } else {
            for (int r = threadIdx.x; r < NC; r += kSolveThreads) {
                const int cj = r / (S::TX / 2), ci = r - cj * (S::TX / 2);
                const int I = i0 / 2 + ci, J = j0 / 2 + cj;
                if (I >= C.nx || J >= C.ny) continue;
                const int ri = HALO + 2 * ci, rj = HALO + 2 * cj;
                const double a = tile_residual<S>(L, H.coef, t, ri, rj, unit);
                const double b = tile_residual<S>(L, H.coef, t, ri + 1, rj, unit);
                const double c = tile_residual<S>(L, H.coef, t, ri, rj + 1, unit);
                const double d = tile_residual<S>(L, H.coef, t, ri + 1, rj + 1, unit);
                C.b[J * C.nx + I] = 0.25 * (a + b + c + d);
            }
        }
        __syncthreads();
    }
}

// up phase of level l: x + prolong(x_coarse) * mask, then the two reverse sweeps
// (solvers_var.py:148-150). With H.fused_res, level 0's tiles are one NumPy leaf
// per interior row (128 cells starting at a multiple of 128): after the sweeps
// every interior cell and its four neighbours hold the new x, so each warp forms
// the squared residual (b - A x)^2 of one row and its leaf sum in NumPy's order
// -- the per-cycle residual norm without another pass over the grid.
template <class S>
__device__ __noinline__ void mg_up(int l, const double* xin, double* xout, int smem, int persist) {
    const HelmParams& H = s_helm;
    double* leaves = (l == 0 && H.fused_res) ? H.leafA : nullptr;
    const double* xc = H.lv[l + 1].x2;  // the coarser level's final x
    const int cnx = H.lv[l + 1].nx;
    const HLevel& L = H.lv[l];
    const bool unit = H.unit_mask != 0;
    const int tx = (L.nx + S::TX - 1) / S::TX, ty = (L.ny + S::TY - 1) / S::TY;
    const bool keep = persist >= 0;
    const TileRefs t = tile_arrays<S>(smem, persist);
    for (int tile = keep ? level0_tile_of_cta(tx * ty) : first_tile(tx * ty); tile < tx * ty; tile += s_grid.ncta) {
        if (tile < 0) continue;  // CTA-uniform: this CTA holds no persistent tile
        const int i0 = (tile % tx) * S::TX, j0 = (tile / tx) * S::TY;
        if (!keep) tile_load<S, true>(L, i0, j0, xin, xc, cnx, t);
        else if constexpr (S::TX == TileWide::TX) {
            if (H.keep_x0) tile_refresh<S>(L, i0, j0, xin, xc, cnx, t);
            else tile_load<S, false>(L, i0, j0, xin, xc, cnx, t);
        }
        tile_four_half_sweeps<S>(L, t, 1, unit);
        tile_store_x<S>(L, i0, j0, t, xout);
        if constexpr (S::TX == 128) {
            if (leaves) {
                const int lane = threadIdx.x & 31;
                // a warp's row of squares, above the tile
                double* row = smem_all + smem + (keep ? (H.keep_x0 ? 0 : 2 * S::SN) : 6 * S::SN) + (threadIdx.x >> 5) * kLeafRow;
                for (int cj = threadIdx.x >> 5; cj < S::TY; cj += kSolveThreads / 32) {
                    if (j0 + cj >= L.ny) continue;  // warp-uniform
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const double d = tile_residual<S>(L, H.coef, t, HALO + lane + 32 * q, cj + HALO, unit);
                        row[lane + 32 * q] = d * d;
                    }
                    __syncwarp();
                    const double a = leaf_sums(row, row, 128).x;
                    if (lane == 0) leaves[H.leaf_slot[((j0 + cj) * L.nx + i0) / 128]] = a;
                    __syncwarp();
                }
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ coarse levels in one CTA
// The levels [coarse_from, n_levels) in one CTA's shared memory: ku, kv, id and m of all
// of them, then x and b, then the scratch of the restriction (one value per cell of the
// first). `coef` is where the four coefficient arrays are when they stand apart, else -1. Even-sized levels store their colours apart: cell
// (i, j) of colour p at [p][j][i / 2]. What a level's phases need of its geometry and
// of where its arrays are stands in a table made once per solve (coarse_tab_init): a
// phase is a few hundred cycles long, and finding its arrays level by level and
// dividing by the row length took most of it.
struct CoarseTab {
    int nx, ny, n, even;
    int hx, nh;              // cells of one colour, per row and in all
    unsigned hmag, nmag;     // q / hx and e / nx as high products (0: the divisor is 1)
    int ku, kv, id, m, x, b; // in smem_all
    double cx, cy, dx2, dy2;
};
static constexpr int kCoarseLevels = 8;
static __shared__ CoarseTab s_ct[kCoarseLevels];
static __shared__ int s_cres, s_clevels;
// whether the coarse levels' coefficients stay in place for the solve: in CTA 0's unused
// level-0 region (H.coarse_persist), or behind the working arrays when CTA 0 has no tile of any level
static __shared__ int s_coarse_held;
static constexpr int kFoldScratch = 64;  // a fold's, where the working arrays start

// where the coarse levels' coefficients stand in a grid-wide solve
__device__ __forceinline__ int coarse_coef_at(const HelmParams& H, int base, int persist) {
    if (H.coarse_persist) return persist;
    int work = H.lv[H.coarse_from].n;
    for (int l = H.coarse_from; l < H.n_levels; ++l) work += 2 * H.lv[l].n;
    return base + (work > kFoldScratch ? work : kFoldScratch);
}

__device__ __forceinline__ bool coarse_hold(const HelmParams& H) {
    if (H.coarse_persist) return true;
    if (H.kind != HK_MULTIGRID || H.big_fold || H.coarse_from == 0) return false;
    for (int l = 0; l < H.coarse_from; ++l)
        if (level_tiles(H.lv[l]) >= s_grid.ncta) return false;
    return true;
}

__device__ __forceinline__ int fast_div(int q, unsigned magic) { return magic ? (int)__umulhi((unsigned)q, magic) : q; }

__device__ __noinline__ void coarse_tab_init(int base, int coef) {
    const HelmParams& H = s_helm;
    const int cf = H.coarse_from, nl = H.n_levels - cf;
    if (threadIdx.x < nl) {
        int off = 0, tot = 0;
        for (int q = 0; q < nl; ++q) {
            if (q < (int)threadIdx.x) off += H.lv[cf + q].n;
            tot += H.lv[cf + q].n;
        }
        const HLevel& L = H.lv[cf + threadIdx.x];
        CoarseTab& T = s_ct[threadIdx.x];
        auto magic = [](int d) { return d > 1 ? (unsigned)((0x100000000ULL + d - 1) / d) : 0u; };
        T.nx = L.nx;
        T.ny = L.ny;
        T.n = L.n;
        T.even = ((L.nx | L.ny) & 1) == 0;
        T.hx = L.nx >> 1;
        T.nh = L.n >> 1;
        T.hmag = magic(T.hx);
        T.nmag = magic(L.nx);
        const int cb = coef >= 0 ? coef : base, xb = coef >= 0 ? base : base + 4 * tot;
        T.ku = cb + off;
        T.kv = cb + tot + off;
        T.id = cb + 2 * tot + off;
        T.m = cb + 3 * tot + off;
        T.x = xb + off;
        T.b = xb + tot + off;
        T.cx = L.cx;
        T.cy = L.cy;
        T.dx2 = L.dx2;
        T.dy2 = L.dy2;
        if (threadIdx.x == 0) {
            s_cres = xb + 2 * tot;
            s_clevels = nl;
            s_coarse_held = coarse_hold(H);
        }
    }
    __syncthreads();
}

// position of cell (i, j) in a level's arrays
__device__ __forceinline__ int coarse_pos(const CoarseTab& T, int i, int j) {
    return T.even ? ((i + j) & 1) * T.nh + j * T.hx + (i >> 1) : j * T.nx + i;
}

// the coarse levels' coefficients (asynchronous copies; the caller waits for them
// before its next CTA barrier)
__device__ __noinline__ void coarse_coef_load() {
    const HelmParams& H = s_helm;
    for (int l = 0; l < s_clevels; ++l) {
        const HLevel& L = H.lv[H.coarse_from + l];
        const CoarseTab& T = s_ct[l];
        const int n = T.n;
        for (int e = threadIdx.x; e < n; e += kSolveThreads) {
            const int j = fast_div(e, T.nmag), o = coarse_pos(T, e - j * T.nx, j);
            cpa_ca8(smem_all + T.ku + o, L.Ku + e);
            cpa_ca8(smem_all + T.kv + o, L.Kv + e);
            cpa_ca8(smem_all + T.id + o, L.idm + e);
            cpa_ca8(smem_all + T.m + o, L.mask + e);
        }
    }
}

// positions, in the other colour's arrays, of the four neighbours of cell q of colour p
// of an even level
struct CoarseNbr {
    int e, w, n, s;
};
__device__ __forceinline__ CoarseNbr coarse_nbr(int hx, int nh, unsigned hmag, int p, int q) {
    const int j = fast_div(q, hmag), c = q - j * hx;
    const int s = (p + j) & 1;  // an odd column: the west neighbour has the same half index
    CoarseNbr o;
    o.w = s ? q : (c == 0 ? q - 1 + hx : q - 1);
    o.e = s ? (c + 1 == hx ? q + 1 - hx : q + 1) : q;
    o.n = q + hx >= nh ? q + hx - nh : q + hx;
    o.s = q - hx < 0 ? q - hx + nh : q - hx;
    return o;
}

// barrier of the first `nw` warps of the CTA (those that work on a small level)
__device__ __forceinline__ void warps_sync(int nw) {
    if (nw == 1) __syncwarp();
    else asm volatile("bar.sync 1, %0;" ::"r"(nw * 32) : "memory");
}

// (b - A x) at cell q of colour p of an even level, masked by the caller's choice: with
// `masked` times the mask (the restricted residual), else as the stopping test takes it
__device__ __forceinline__ double coarse_residual(const CoarseTab& T, double coef, bool unit, int p, int q, bool masked) {
    const int nh = T.nh, op = p * nh, oo = nh - op;
    const CoarseNbr o = coarse_nbr(T.hx, nh, T.hmag, p, q);
    const double *x = smem_all + T.x, *ku = smem_all + T.ku, *kv = smem_all + T.kv, *mk = smem_all + T.m;
    const double m = mk[op + q];
    double xm = x[op + q], xe = x[oo + o.e], xw = x[oo + o.w], xn = x[oo + o.n], xs = x[oo + o.s];
    if (!unit) {
        xm = xm * m;
        xe = xe * mk[oo + o.e];
        xw = xw * mk[oo + o.w];
        xn = xn * mk[oo + o.n];
        xs = xs * mk[oo + o.s];
    }
    const double fx = ku[op + q] * (xe - xm);
    const double fxw = ku[oo + o.w] * (xm - xw);
    const double fy = kv[op + q] * (xn - xm);
    const double fys = kv[oo + o.s] * (xm - xs);
    const double lap = (fx - fxw) / T.dx2 + (fy - fys) / T.dy2;
    const double r = smem_all[T.b + op + q] - ((xm - coef * lap) * m + xm * (1.0 - m));
    return masked ? r * m : r;
}

// Four half-sweeps (colours c0, 1 - c0, c0, 1 - c0) of even level l, then, with_res, the
// masked residual of every cell into the scratch (in the level's own order). CPT: cells
// of a colour per thread at most. With one, each thread keeps its cell of either
// colour -- the neighbours' places, the coefficients and b -- in registers throughout,
// and only the warps that have cells take part in the barriers between half-sweeps.
// With more, a thread forms all its values of a half-sweep before it stores any, so
// that their loads run together.
template <int CPT>
__device__ __noinline__ void coarse_sweeps(int l, int c0, bool with_res) {
    const CoarseTab& T = s_ct[l];
    const bool unit = s_helm.unit_mask != 0;
    const double coef = s_helm.coef;
    const int hx = T.hx, nh = T.nh;
    const unsigned hmag = T.hmag;
    const double cx = T.cx, cy = T.cy;
    double* x = smem_all + T.x;
    const double *b = smem_all + T.b, *ku = smem_all + T.ku, *kv = smem_all + T.kv, *id = smem_all + T.id,
                 *mk = smem_all + T.m;
    if constexpr (CPT > 1) {
#pragma unroll 1
        for (int h = 0; h < 4; ++h) {
            const int p = (c0 + h) & 1, op = p * nh, oo = nh - op;
            double v[CPT];
#pragma unroll
            for (int r = 0; r < CPT; ++r) {
                const int q = threadIdx.x + r * kSolveThreads;
                v[r] = 0.0;
                if (q < nh) {
                    const CoarseNbr o = coarse_nbr(hx, nh, hmag, p, q);
                    const double nb = cx * (ku[op + q] * x[oo + o.e] + ku[oo + o.w] * x[oo + o.w]) +
                                      cy * (kv[op + q] * x[oo + o.n] + kv[oo + o.s] * x[oo + o.s]);
                    v[r] = id[op + q] * (b[op + q] + nb);
                    if (!unit) v[r] = v[r] * mk[op + q];
                }
            }
#pragma unroll
            for (int r = 0; r < CPT; ++r) {
                const int q = threadIdx.x + r * kSolveThreads;
                if (q < nh) x[op + q] = v[r];
            }
            __syncthreads();
        }
        if (with_res)
            for (int f = threadIdx.x; f < T.n; f += kSolveThreads) {
                const int p = f >= nh;
                smem_all[s_cres + f] = coarse_residual(T, coef, unit, p, f - p * nh, true);
            }
    } else {
        const int q = threadIdx.x, nw = (nh + 31) >> 5;
        if (q < nw * 32) {
            const bool on = q < nh;
            // index 0: the cell of colour c0, 1: that of the other colour
            CoarseNbr o[2];
            double ke[2], kw[2], kn[2], ks[2], di[2], bb[2];
            if (on) {
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const int p = c0 ^ a, op = p * nh, oo = nh - op;
                    o[a] = coarse_nbr(hx, nh, hmag, p, q);
                    ke[a] = ku[op + q];
                    kw[a] = ku[oo + o[a].w];
                    kn[a] = kv[op + q];
                    ks[a] = kv[oo + o[a].s];
                    di[a] = id[op + q];
                    bb[a] = b[op + q];
                }
            }
#pragma unroll 1
            for (int r = 0; r < 2; ++r) {
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    if (on) {
                        const int op = (c0 ^ a) * nh;
                        const double* xo = x + (nh - op);
                        const double nb = cx * (ke[a] * xo[o[a].e] + kw[a] * xo[o[a].w]) +
                                          cy * (kn[a] * xo[o[a].n] + ks[a] * xo[o[a].s]);
                        double v = di[a] * (bb[a] + nb);
                        if (!unit) v = v * mk[op + q];
                        x[op + q] = v;
                    }
                    warps_sync(nw);
                }
            }
            if (with_res && on) {
#pragma unroll
                for (int p = 0; p < 2; ++p) smem_all[s_cres + p * nh + q] = coarse_residual(T, coef, unit, p, q, true);
            }
        }
    }
    __syncthreads();
}

// the same sweeps of an odd-sized (coarsest) level in the flat order, each cell tested for its colour
__device__ __noinline__ void coarse_sweeps_odd(int l, int c0) {
    const CoarseTab& T = s_ct[l];
    const bool unit = s_helm.unit_mask != 0;
    const int nx = T.nx, ny = T.ny;
    double* x = smem_all + T.x;
    const double *b = smem_all + T.b, *ku = smem_all + T.ku, *kv = smem_all + T.kv, *id = smem_all + T.id;
    for (int h = 0; h < 4; ++h) {
        const int colour = (c0 + h) & 1;
        for (int e = threadIdx.x; e < T.n; e += kSolveThreads) {
            const int j = fast_div(e, T.nmag), i = e - j * nx;
            if (((i + j) & 1) != colour) continue;
            const int ie = i + 1 == nx ? e + 1 - nx : e + 1, iw = i == 0 ? e - 1 + nx : e - 1;
            const int jn = j + 1 == ny ? i : e + nx, js = j == 0 ? e + T.n - nx : e - nx;
            const double nb = T.cx * (ku[e] * x[ie] + ku[iw] * x[iw]) + T.cy * (kv[e] * x[jn] + kv[js] * x[js]);
            double v = id[e] * (b[e] + nb);
            if (!unit) v = v * smem_all[T.m + e];
            x[e] = v;
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void coarse_level_sweeps(int l, int c0, bool with_res) {
    const int even = s_ct[l].even, nh = s_ct[l].nh;
    if (!even) coarse_sweeps_odd(l, c0);
    else if (nh > kSolveThreads) coarse_sweeps<(kOneCtaCells / 2 + kSolveThreads - 1) / kSolveThreads>(l, c0, with_res);
    else coarse_sweeps<1>(l, c0, with_res);
}

// The V-cycle on the levels from coarse_from on by one CTA, x and b of the first of
// them in place in shared memory (and its coefficients and those below).
__device__ __noinline__ void coarse_cycle() {
    const int nl = s_clevels;
    for (int l = 0; l < nl; ++l) {
        coarse_level_sweeps(l, 0, l + 1 < nl);
        if (l + 1 < nl) {
            // a coarser level exists only below an even-sized one: its cells are exactly
            // the 2 x 2 children, and the residual's mean over them is its right-hand side
            const CoarseTab &F = s_ct[l], &C = s_ct[l + 1];
            const int nh = F.nh, hx = F.hx;
            const double* res = smem_all + s_cres;
            for (int e = threadIdx.x; e < C.n; e += kSolveThreads) {
                const int J = fast_div(e, C.nmag), I = e - J * C.nx;
                // children (2I, 2J), (2I+1, 2J), (2I, 2J+1), (2I+1, 2J+1): colours 0, 1, 1, 0
                const int r0 = 2 * J * hx + I, r1 = r0 + hx;
                const int o = coarse_pos(C, I, J);
                smem_all[C.b + o] = 0.25 * (res[r0] + res[nh + r0] + res[nh + r1] + res[r1]);
                smem_all[C.x + o] = 0.0;
            }
            __syncthreads();
        }
    }
    // the coarsest level: its reverse sweeps follow the forward ones directly
    coarse_level_sweeps(nl - 1, 1, false);
    for (int l = nl - 2; l >= 0; --l) {
        const CoarseTab &F = s_ct[l], &C = s_ct[l + 1];
        // x + prolong(e) mask on colour 0, the cells the first reverse half-sweep (of
        // colour 1) reads; colour 1's own x is overwritten without being read
        double* x = smem_all + F.x;
        for (int q = threadIdx.x; q < F.nh; q += kSolveThreads) {
            const int j = fast_div(q, F.hmag), I = q - j * F.hx;
            x[q] = x[q] + smem_all[C.x + coarse_pos(C, I, j >> 1)] * smem_all[F.m + q];
        }
        __syncthreads();
        coarse_level_sweeps(l, 1, false);
    }
}

// the coarse levels of a larger grid, by CTA 0: level cf's b from global memory and its
// x back; the table is made (coarse_tab_init), and the coefficients are in place when
// they persist for the solve
__device__ __noinline__ void mg_coarse(const double* xin_cf, double* xout_cf, bool load_coef) {
    const HelmParams& H = s_helm;
    const CoarseTab& T = s_ct[0];
    const double* b = H.lv[H.coarse_from].b;
    if (load_coef) coarse_coef_load();
    for (int e = threadIdx.x; e < T.n; e += kSolveThreads) {
        const int j = fast_div(e, T.nmag), o = coarse_pos(T, e - j * T.nx, j);
        const double bv = __ldcg(b + e);
        smem_all[T.x + o] = xin_cf ? __ldcg(xin_cf + e) : 0.0;
        smem_all[T.b + o] = bv;
    }
    cpa_wait_all();
    __syncthreads();
    coarse_cycle();
    for (int e = threadIdx.x; e < T.n; e += kSolveThreads) {
        const int j = fast_div(e, T.nmag);
        xout_cf[e] = smem_all[T.x + coarse_pos(T, e - j * T.nx, j)];
    }
    __syncthreads();
}

// ------------------------------------------------------------------ the coarsest level on the grid
__device__ __forceinline__ bool level_even(const HLevel& L) { return ((L.nx | L.ny) & 1) == 0; }

// The region of an odd-sized level's tile in the flat order; all of a thread's loads are
// issued before its first store to shared memory. code[k] is twice the ring of the
// thread's k-th cell plus its colour, which the grid coordinates give (-1: no cell).
static constexpr int kFlatCells = (Tile32::RN + kSolveThreads - 1) / kSolveThreads;
__device__ __forceinline__ void flat_load(const HLevel& L, int i0, int j0, const double* xin, TileRefs t,
                                          int (&code)[kFlatCells]) {
    constexpr int RW = Tile32::RW, RH = Tile32::RH;
    double xv[kFlatCells], bv[kFlatCells];
#pragma unroll
    for (int k = 0; k < kFlatCells; ++k) {
        const int r = threadIdx.x + k * kSolveThreads;
        xv[k] = bv[k] = 0.0;
        code[k] = -1;
        if (r >= Tile32::RN) continue;
        const int rj = r / RW, ri = r - rj * RW;
        const int gi = wrap_any(i0 - HALO + ri, L.nx), gj = wrap_any(j0 - HALO + rj, L.ny);
        const int g = gj * L.nx + gi;
        code[k] = 2 * min(min(ri, RW - 1 - ri), min(rj, RH - 1 - rj)) + ((gi + gj) & 1);
        cpa_ca8(t.ku + r, L.Ku + g);
        cpa_ca8(t.kv + r, L.Kv + g);
        cpa_ca8(t.id + r, L.idm + g);
        cpa_ca8(t.m + r, L.mask + g);
        if (xin) xv[k] = __ldcg(xin + g);
        bv[k] = __ldcg(L.b + g);
    }
#pragma unroll
    for (int k = 0; k < kFlatCells; ++k) {
        const int r = threadIdx.x + k * kSolveThreads;
        if (r >= Tile32::RN) continue;
        t.x[r] = xv[k];
        t.b[r] = bv[k];
    }
    cpa_wait_all();
    __syncthreads();
}

// a half-sweep of such a tile: the cells of colour `colour` on the rings from `ring` on
__device__ __forceinline__ void flat_half_sweep(const HLevel& L, TileRefs t, const int (&code)[kFlatCells], int ring,
                                                int colour, bool unit) {
    constexpr int RW = Tile32::RW;
#pragma unroll
    for (int k = 0; k < kFlatCells; ++k) {
        if (code[k] < 2 * ring || (code[k] & 1) != colour) continue;
        const int r = threadIdx.x + k * kSolveThreads;
        const double nb = L.cx * (t.ku[r] * t.x[r + 1] + t.ku[r - 1] * t.x[r - 1]) +
                          L.cy * (t.kv[r] * t.x[r + RW] + t.kv[r - RW] * t.x[r - RW]);
        double v = t.id[r] * (t.b[r] + nb);
        if (!unit) v = v * t.m[r];
        t.x[r] = v;
    }
    __syncthreads();
}

// Smoothing of a coarsest level too large for CTA 0: two forward or two reverse sweeps on
// 32 x 32 tiles, colours apart where the level is even. us a solve with all tiles in the flat
// order, loaded cell by cell and each cell's colour worked out in every sweep, and so:
// 1000 x 10 199 and 170, 75 x 75 218 and 188, 257 x 129 223 and 196.
__device__ __noinline__ void mg_smooth(int l, const double* xin, double* xout, bool reverse, int smem) {
    using S = Tile32;
    const HelmParams& H = s_helm;
    const HLevel& L = H.lv[l];
    const bool unit = H.unit_mask != 0;
    const int tx = (L.nx + S::TX - 1) / S::TX, ty = (L.ny + S::TY - 1) / S::TY;
    const TileRefs t = tile_arrays<S>(smem, -1);
    const int c0 = reverse ? 1 : 0;
    const bool even = level_even(L);
    for (int tile = s_grid.cta; tile < tx * ty; tile += s_grid.ncta) {
        const int i0 = (tile % tx) * S::TX, j0 = (tile / tx) * S::TY;
        if (even) {
            tile_load<S, true>(L, i0, j0, xin, nullptr, 0, t);
            tile_four_half_sweeps<S>(L, t, c0, unit);
            tile_store_x<S>(L, i0, j0, t, xout);
        } else {
            int code[kFlatCells];
            flat_load(L, i0, j0, xin, t, code);
#pragma unroll 1
            for (int h = 0; h < 4; ++h) flat_half_sweep(L, t, code, h + 1, (c0 + h) & 1, unit);
            for (int r = threadIdx.x; r < S::TX * S::TY; r += kSolveThreads) {
                const int cj = r / S::TX, ci = r - cj * S::TX;
                const int gi = i0 + ci, gj = j0 + cj;
                if (gi >= L.nx || gj >= L.ny) continue;
                xout[gj * L.nx + gi] = t.x[(cj + HALO) * S::RW + ci + HALO];
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ the cycle
// one V(2,2) cycle on x0 (level 0's current x); returns the buffer holding the
// new x (x0 or level 0's second buffer). Levels below coarse_from have a grid
// down and up phase; the rest run in CTA 0, or, when every level is too large
// for it, the coarsest level is smoothed on the grid.
// work0 runs beside level 0's down phase, which only reads x0, and stop0 after the
// barrier that ends that phase: where it returns true the cycle is given up and x0 is
// the result.
template <class W, class S>
__device__ __forceinline__ double* vcycle_tiled(const HelmParams& H, double* x0, double* x0b, int smem, int persist,
                                                bool& ok, W work0, S stop0) {
    const int cf = H.coarse_from, nl = H.n_levels;
    if (cf == 0) {
        if (s_grid.cta == 0) mg_coarse(x0, x0b, true);
        ok = grid_sync(H);
        return x0b;
    }
    const int ndown = cf < nl ? cf : nl - 1;
    for (int l = 0; l < ndown && ok; ++l) {
        const double* xin = l == 0 ? x0 : nullptr;
        double* xout = l == 0 ? x0b : H.lv[l].x;
        switch (H.lv[l].shape) {
            case SHAPE_WIDE: mg_down<TileWide>(l, xin, xout, smem, l == 0 ? persist : -1); break;
            case SHAPE_3216: mg_down<Tile3216>(l, xin, xout, smem, -1); break;
            case SHAPE_16: mg_down<Tile16>(l, xin, xout, smem, -1); break;
            case SHAPE_8: mg_down<Tile8>(l, xin, xout, smem, -1); break;
            default: mg_down<Tile32>(l, xin, xout, smem, -1); break;
        }
        if (l == 0) work0();
        ok = grid_sync(H);
        if (l == 0 && ok && stop0()) return x0;
    }
    if (!ok) return x0;
    if (cf < nl) {
        if (s_grid.cta == 0) mg_coarse(nullptr, H.lv[cf].x2, !s_coarse_held);
        ok = grid_sync(H);
    } else {
        const int l = nl - 1;
        double* xa = (l == 0) ? x0b : H.lv[l].x;
        double* xb = (l == 0) ? x0 : H.lv[l].x2;
        mg_smooth(l, l == 0 ? x0 : nullptr, xa, false, smem);
        ok = grid_sync(H);
        if (!ok) return x0;
        mg_smooth(l, xa, xb, true, smem);
        ok = grid_sync(H);
        if (l == 0) return x0;
    }
    // ascend: level l reads its down-phase result and level l+1's final x (in x2)
    for (int l = ndown - 1; l >= 0 && ok; --l) {
        const double* xin = (l == 0) ? x0b : H.lv[l].x;
        double* xout = (l == 0) ? x0 : H.lv[l].x2;
        switch (H.lv[l].shape) {
            case SHAPE_WIDE: mg_up<TileWide>(l, xin, xout, smem, l == 0 ? persist : -1); break;
            case SHAPE_3216: mg_up<Tile3216>(l, xin, xout, smem, -1); break;
            case SHAPE_16: mg_up<Tile16>(l, xin, xout, smem, -1); break;
            case SHAPE_8: mg_up<Tile8>(l, xin, xout, smem, -1); break;
            default: mg_up<Tile32>(l, xin, xout, smem, -1); break;
        }
        ok = grid_sync(H);
    }
    return x0;
}

}  // namespace oc
