// Column and stencil kernels of the ocean-core step (sm_100a, fp64).
//
// The column kernels map one thread to one water column (i, j) and march over
// the levels k, so every vertical recurrence of the reference (cumulative sums,
// Thomas sweeps, the closure's mixing-length marches) runs in the reference's
// order; the 32 threads of a warp read 32 consecutive i of each level plane
// (coalesced 256-byte rows). The stencil kernels (k_mom_column, k_tracer_rhs,
// k_predictor_rhs) work on tiles of columns over a range of levels.
//
// Reference correspondence (paths inside the reference project):
//   k_closure         libs/core/closure.py:43-205 + model3d_v05.py:141-157 (q = A^-1 1)
//   k_qsolve          model3d_v05.py:147-153 (constant-coefficient q)
//   k_kukv            model3d_v05.py:154-157
//   k_wcol            vertical_var.py:109-121 + model3d_v05.py:232-235
//   k_phi             vertical_var.py:132-145
//   k_mom_column      model3d_v05.py:195-230, 241-260, 352-370; advection_v06.py:77-108;
//                     advection.py:62-95; operators_masked.py:45-68; vertical_var.py:80-106
//   k_predictor_rhs   model3d_v05.py:387-393
//   k_momentum_solve  model3d_v05.py:394-395, 426-433 + vertical.py:17-44
//   k_backsub         model3d_v05.py:404-406
//   k_tracer_rhs      model3d_v05.py:466-512
//   k_tracer_solve    model3d_v05.py:514-533 + eos.py:68-133
//   2D kernels        model3d_v05.py:290-335, 376-384, 396-400, 410-413, 440-461

#include <algorithm>
#include <atomic>

#include "oc_internal.cuh"
#include "step_common.cuh"
#include "step_kernels.cuh"

namespace oc {

// The floating type of the 3D fields: double for the fp64 path, float for the
// mixed-precision path (OC_MIXED builds this file a second time). The buoyancy
// b and the buoyancy potential phi stay fp64 on both paths (wide), and so do
// every 2D field and every depth-integrated sum.
#ifdef OC_MIXED
typedef float real;
#else
typedef double real;
#endif
typedef double wide;

// Minimum resident CTAs per SM the register allocation of the three largest
// stencil/column kernels is bounded for (__launch_bounds__): k_closure runs
// 128 threads, k_mom_column 512 and k_tracer_rhs 256 per CTA. The bits of the
// results do not depend on them.
#ifndef OC_MINB_CLOSURE
#ifdef OC_MIXED
#define OC_MINB_CLOSURE 4
#else
#define OC_MINB_CLOSURE 8
#endif
#endif
#ifndef OC_MINB_MOM
#define OC_MINB_MOM 2
#endif
#ifndef OC_MINB_TRACER
#ifdef OC_MIXED
#define OC_MINB_TRACER 6  // FP32: 0.56 against 0.59 ms per step at 512 x 512 x 50
#else
#define OC_MINB_TRACER 4
#endif
#endif
using KPR = KPT<real>;
using KLR = KLT<real>;  // with the level table
using ColGeoR = ColGeoT<real>;

// ------------------------------------------------------------------ helpers



__device__ __forceinline__ real m3u_at(const KPR& P, const Nbr& n, int dj, int di, int k) {
    return col_m3u(P, n.at(dj, di), k);
}

__device__ __forceinline__ real m3v_at(const KPR& P, const Nbr& n, int dj, int di, int k) {
    return col_m3v(P, n.at(dj, di), k);
}

__device__ __forceinline__ real m3_at(const KPR& P, const Nbr& n, int dj, int di, int k) {
    return col_m3(P, n.at(dj, di), k);
}



// ------------------------------------------------------------------ q = A^-1 1 on a column
// interface spacing of the column (closure.py:43-62): dz[0] at the surface,
// dz[nz-1] at the bottom, the mean of the two levels elsewhere
__device__ __forceinline__ real col_dzi(const KLR& P, const ColGeoR& g, int k) {
    if (k < g.kf) return P.dzi[k];
    real m;
    if (k == 0) return g.dz(P, 0, m);
    if (k == P.nz) return g.dz(P, P.nz - 1, m);
    const real a = g.dz(P, k - 1, m);
    return real(0.5) * (a + g.dz(P, k, m));
}

// Momentum tridiagonal with a unit right-hand side for the column's interface
// viscosity Km(k), k = 0..nz (reference model3d_v05.py:147-153). The forward
// elimination keeps its coefficients in cs and its right-hand sides in q, which
// the back substitution then overwrites with the solution.
template <class KM>
__device__ __forceinline__ void column_q(const KLR& P, const ColGeoR& g, KM Km, real* cs,
                                         real* __restrict__ q, int c, size_t n2) {
    const int nz = P.nz;
    real rdzi_k = g.rdz(P, 0);
    real km_k = Km(0);
    real ds = real(0.0), cp = real(0.0);
#pragma unroll 2
    for (int k = 0; k < nz; ++k) {
        const real m3_k = k < g.kb ? real(1.0) : real(0.0), m3_k1 = k + 1 < g.kb ? real(1.0) : real(0.0);
        const real rdzi_k1 = (k + 1 < nz) ? g.rdzi(P, k + 1) : real(0.0);
        const real km_k1 = Km(k + 1);
        real sub, diag, sup;
        implicit_row_inv(P, k, g.rdz(P, k), m3_k, m3_k1, rdzi_k, rdzi_k1, km_k, km_k1, P.thv_dt_drag, sub, diag, sup);
        if (k == 0) {
            cp = sup / diag;
            ds = real(1.0) / diag;
        } else {
            const real den = diag - sub * cp;
            cp = sup / den;
            ds = (real(1.0) - sub * ds) / den;
        }
        cs[k] = cp;
        if (k + 1 < nz) q[(size_t)k * n2 + c] = ds;
        km_k = km_k1;
        rdzi_k = rdzi_k1;
    }
    real x = ds;
    q[(size_t)(nz - 1) * n2 + c] = x;
#pragma unroll 4
    for (int k = nz - 2; k >= 0; --k) {
        const size_t o = (size_t)k * n2 + c;
        x = q[o] - cs[k] * x;
        q[o] = x;
    }
}

template <int NZM>
__global__ void __launch_bounds__(128) k_qsolve(KLR P, const real* __restrict__ km,
                                                real* __restrict__ q) {
    COLUMN_PROLOGUE
    const int c = nb.c;
    const ColGeoR g = ColGeoR::load(P, c);
    real cs[NZM];
    column_q(P, g, [&](int k) { return km[(size_t)k * n2 + c]; }, cs, q, c, n2);
}

// ------------------------------------------------------------------ TKE closure
// One thread per column (closure.py:141-205): shear and N^2 on interfaces, the
// mixing lengths, the implicit TKE tridiagonal (nz+1 rows), K_m/K_h, then q for
// the new K_m. With the Gaspar lengths, the lengths of interface k are formed inside
// the forward sweep. Per thread only N^2, shear^2 and column_q's elimination
// coefficients are kept: an array per thread is in local memory, which at 512 x 512 does
// not fit the caches (1.5 KB a column), while e, q and kh are there anyway -- the
// elimination's right-hand sides go to e (whose old value at a level is read just
// before), its coefficients to q, the mixing lengths to kh until K_h replaces them.
// Reciprocals of full columns' thicknesses and spacings come from the level table.
// 512 x 512 x 50: 817 us a launch before, 750 now (FP32 542 and 465); fewer CTAs per SM
// make it slower, so its loads' latency bounds it, not the caches' size.
template <int NZM>
__global__ void __launch_bounds__(128, OC_MINB_CLOSURE) k_closure(KLR P, const real* __restrict__ u,
                                                 const real* __restrict__ v,
                                                 const wide* __restrict__ b,
                                                 real* __restrict__ e, real* __restrict__ km,
                                                 real* __restrict__ kh, real* __restrict__ q) {
#ifdef OC_MIXED
    // FP32 build: N^2 of the column on its interfaces, which the Gaspar length
    // marches read O(nz) times per interface, lives in shared memory: interface k
    // of the CTA's thread t at [k * threads + t] (dynamic, (nz + 1) x threads
    // values). Measured at 512 x 512 x 50: 0.52 against 0.57 ms for the local
    // array; the fp64 build keeps the local array (0.81 against 1.07 ms).
    extern __shared__ __align__(16) unsigned char s_dyn[];
    const StridedCol<real> nn2{reinterpret_cast<real*>(s_dyn) + threadIdx.y * blockDim.x + threadIdx.x,
                               (int)(blockDim.x * blockDim.y)};
#endif
    COLUMN_PROLOGUE
    const int nz = P.nz;
    const int c = nb.c;
    const size_t cw = nb.at(0, -1), cs_ = nb.at(-1, 0);
    const ColGeoR g = ColGeoR::load(P, c);
#ifndef OC_MIXED
    real nn2[NZM + 1];
#endif
    real le[NZM + 1], cst[NZM];
    real sh2[NZM + 1];
    real depth = real(0.0);
    for (int k = 0; k < nz; ++k) {
        real m;
        const real dz = g.dz(P, k, m);
        depth = (k == 0) ? dz : depth + dz;
    }
    // shear^2 and N^2 on interfaces (closure.py:150-161)
    {
        real uc_prev = real(0.0), vc_prev = real(0.0);
        wide b_prev = 0.0;
#pragma unroll 2
        for (int k = 0; k < nz; ++k) {
            const size_t o = (size_t)k * n2;
            const real uc = real(0.5) * (u[o + c] + u[o + cw]);
            const real vc = real(0.5) * (v[o + c] + v[o + cs_]);
            const wide bk = b[o + c];
            if (k >= 1) {
                const real wk = k < g.kb ? real(1.0) : real(0.0);
                const real idz = g.rdzi(P, k);
                const real du = (uc_prev - uc) * idz;
                const real dv = (vc_prev - vc) * idz;
                sh2[k] = (du * du + dv * dv) * wk;
                // the difference of two fp64 buoyancies (their ~1e-2 relative
                // vertical contrast would lose digits in FP32)
                const real db = real((b_prev - bk) * idz);
                nn2[k] = db * wk;
            }
            uc_prev = uc;
            vc_prev = vc;
            b_prev = bk;
        }
    }
    sh2[0] = real(0.0);
    sh2[nz] = real(0.0);
    nn2[0] = real(0.0);
    nn2[nz] = real(0.0);
    // recursive lengths (closure.py:106-129) need whole-column sweeps first
    if (P.mxl_recursive) {
        real zi = real(0.0);
        for (int k = 0; k <= nz; ++k) {
            real m;
            if (k >= 1) zi = (k == 1) ? g.dz(P, 0, m) : zi + g.dz(P, k - 1, m);
            const real zb = fmax(depth - zi, real(0.0));
            const real ek = fmax(e[(size_t)k * n2 + c], P.e_min);
            const real n2c = fmax(nn2[k], P.n2_min);
            const real ell = sqrt(real(2.0) * ek / n2c);
            le[k] = fmin(ell, fmin(zi + P.z_0, zb + P.z_0));
        }
        for (int k = 1; k <= nz; ++k) le[k] = fmin(le[k], le[k - 1] + col_dzi(P, g, k));
        for (int k = nz - 1; k >= 0; --k) le[k] = fmin(le[k], le[k + 1] + col_dzi(P, g, k + 1));
    }
    // implicit TKE rows and forward sweep (closure.py:171-198)
    real rhs0 = real(0.0), ds = real(0.0), cp = real(0.0), zi = real(0.0);
    real km_prev = real(0.0), km_cur = km[c];
    real m3_km1 = real(0.0), dz_km1 = real(0.0);  // level k-1
    real m3_k, dz_k = g.dz(P, 0, m3_k);
    for (int k = 0; k <= nz; ++k) {
        const size_t o = (size_t)k * n2 + c;
        const real km_next = (k < nz) ? km[o + n2] : real(0.0);
        const real wk = (k >= 1 && k <= nz - 1) ? m3_km1 * m3_k : real(0.0);
        const real e_old = e[o], kh_old = kh[o];
        const real sh2_k = sh2[k];
        real le_k, lk_k;
        if (!P.mxl_recursive) {
            // Gaspar lengths (closure.py:65-104): march away from interface k
            // until the energy budget is spent; once the budget is zero the
            // reference's remaining steps add exactly 0
            if (k >= 1) zi = (k == 1) ? dz_km1 : zi + dz_km1;
            const real zb = fmax(depth - zi, real(0.0));
            const real ek = fmax(e_old, P.e_min);
            real lu = real(0.0), bud = ek;
            for (int kk = k - 1; kk >= 0 && bud > real(0.0); --kk) {
                const real n2j = fmax(nn2[kk], real(0.0)), dzj = col_dzi(P, g, kk);
                const real cost = n2j * dzj * (lu + real(0.5) * dzj);
                const bool full = cost <= bud;
                real step = dzj;
                if (!full && n2j > real(0.0)) {
                    const real part = sqrt(fmax(lu * lu + real(2.0) * bud / n2j, real(0.0))) - lu;
                    step = fmin(fmax(part, real(0.0)), dzj);
                }
                lu = lu + step;
                bud = full ? bud - cost : real(0.0);
            }
            real ld = real(0.0);
            bud = ek;
            for (int kk = k + 1; kk <= nz && bud > real(0.0); ++kk) {
                const real n2j = fmax(nn2[kk], real(0.0)), dzj = col_dzi(P, g, kk);
                const real cost = n2j * dzj * (ld + real(0.5) * dzj);
                const bool full = cost <= bud;
                real step = dzj;
                if (!full && n2j > real(0.0)) {
                    const real part = sqrt(fmax(ld * ld + real(2.0) * bud / n2j, real(0.0))) - ld;
                    step = fmin(fmax(part, real(0.0)), dzj);
                }
                ld = ld + step;
                bud = full ? bud - cost : real(0.0);
            }
            lu = fmin(lu, zi + P.z_0) * wk;
            ld = fmin(ld, zb + P.z_0) * wk;
            lk_k = fmax(P.l_min, sqrt(lu * ld));
            le_k = fmax(P.l_min, fmin(lu, ld));
        } else {
            const real ell = le[k] * wk;
            lk_k = fmax(P.l_min, sqrt(ell * ell));
            le_k = fmax(P.l_min, fmin(ell, ell));
        }
        kh[o] = lk_k;  // until the back substitution, which turns it into K_h
        const real prod = (km_cur - P.nu) * sh2_k - (kh_old - P.kappa) * nn2[k];
        const real diss = P.c_eps * sqrt(fmax(e_old, P.e_min)) / le_k;
        real a_up = real(0.0), a_dn = real(0.0);
        if (k >= 1 && k <= nz - 1) {
            const real idzi = g.rdzi(P, k);
            a_up = P.dt * (real(0.5) * (km_prev + km_cur)) * g.rdz(P, k - 1) * idzi;
            a_dn = P.dt * (real(0.5) * (km_cur + km_next)) * g.rdz(P, k) * idzi;
        }
        real sub = -a_up, sup = -a_dn;
        real diag = real(1.0) + a_up + a_dn + P.dt * diss;
        real rhs = e_old + P.dt * prod;
        if (wk <= real(0.0)) {
            diag = real(1.0);
            sub = real(0.0);
            sup = real(0.0);
            rhs = P.e_min;
        }
        if (k == 0) {
            rhs = (g.kb > 0) ? P.e_bb * P.ustar2[c] : P.e_min;
            rhs0 = rhs;
            cp = sup / diag;
            ds = rhs / diag;
        } else {
            const real den = diag - sub * cp;
            cp = sup / den;
            ds = (rhs - sub * ds) / den;
        }
        if (k < nz) q[o] = cp;  // the elimination coefficients, until column_q
        e[o] = ds;
        km_prev = km_cur;
        km_cur = km_next;
        m3_km1 = m3_k;
        dz_km1 = dz_k;
        if (k + 1 < nz) {
            dz_k = g.dz(P, k + 1, m3_k);
        } else {
            dz_k = real(0.0);
            m3_k = real(0.0);
        }
    }
    // back substitution, e/K update (closure.py:198-205)
    real x = real(0.0);
    for (int k = nz; k >= 0; --k) {
        const size_t o = (size_t)k * n2 + c;
        x = (k == nz) ? ds : e[o] - q[o] * x;
        real m0, m1;
        g.dz(P, k >= 1 ? k - 1 : 0, m0);
        g.dz(P, k < nz ? k : 0, m1);
        const real wk = (k >= 1 && k <= nz - 1) ? m0 * m1 : real(0.0);
        real en = fmax(x, P.e_min);
        en = (wk > real(0.0)) ? en : P.e_min;
        if (k == 0) en = rhs0;
        const real kmn = P.c_k * kh[o] * sqrt(en) * wk + P.nu;
        const real kx = kmn - P.nu;
        const real khn = (P.pr_t == real(1.0) ? kx : kx / P.pr_t) + P.kappa;
        e[o] = en;
        km[o] = kmn;
        kh[o] = khn;
    }
    column_q(P, g, [&](int k) { return km[(size_t)k * n2 + c]; }, cst, q, c, n2);
}

// The same closure by levels (the Gaspar lengths, which march over the column from each
// interface, take most of its time): a CTA takes CL_X columns of a row with CL_Y threads
// each. The threads form N^2, the lengths and the rows of the column's
// interfaces side by side, in shared memory; the two eliminations are done by one
// thread a column. Values and their operations are k_closure's. For few columns: us a
// launch by columns and by levels, 48 x 48 x 12 9.5 and 3.5, 16,384 x 50 211 and 99, 32,000 x
// 40 96 and 61, with recursive lengths 46,937 x 37 206 and 170; at 262,144 x 50 732 and 938,
// where k_closure has warps enough and the shared arrays leave this one 24 to an SM. Four
// or sixteen threads a column are within 20% of eight.
constexpr int CL_X = 32, CL_Y = 8;
__global__ void __launch_bounds__(CL_X * CL_Y, 3) k_closure_levels(
    KLR P, const real* __restrict__ u, const real* __restrict__ v, const wide* __restrict__ b, real* __restrict__ e,
    real* __restrict__ km, real* __restrict__ kh, real* __restrict__ q) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    const int tiles = (P.nx + CL_X - 1) / CL_X;
    const int j = blockIdx.x / tiles, i_own = (blockIdx.x - j * tiles) * CL_X + threadIdx.x;
    const bool live = i_own < P.nx;  // the others repeat the last column and store nothing
    const int i = live ? i_own : P.nx - 1;
    const int nz = P.nz, nx = P.nx, rows = (nz + 1) * CL_X, first = threadIdx.y;
    const size_t n2 = (size_t)P.n2;
    const int c = j * nx + i, cw = j * nx + wrapi(i - 1, nx), cs_ = wrapi(j - 1, P.ny) * nx + i;
    const ColGeoR g = ColGeoR::load(P, c);
    // of the thread's column, interface k at [k * CL_X]: N^2, then the new K_m; the rows,
    // of which sup becomes the elimination's coefficient and rhs the solution
    real* s_n2 = reinterpret_cast<real*>(s_dyn) + threadIdx.x;
    real *s_sub = s_n2 + rows, *s_dia = s_sub + rows, *s_sup = s_dia + rows, *s_rhs = s_sup + rows;
    auto wet = [&](int k) { return k < g.kb ? real(1.0) : real(0.0); };
    auto inner = [&](int k) { return (k >= 1 && k <= nz - 1) ? wet(k - 1) * wet(k) : real(0.0); };
    // x of the rows: forward elimination, then back, in place
    auto solve = [&](int n) {
        real cp = real(0.0), ds = real(0.0);
#pragma unroll 2
        for (int k = 0; k < n; ++k) {
            const real sub = s_sub[k * CL_X], dia = s_dia[k * CL_X], sup = s_sup[k * CL_X], rhs = s_rhs[k * CL_X];
            if (k == 0) {
                cp = sup / dia;
                ds = rhs / dia;
            } else {
                const real den = dia - sub * cp;
                cp = sup / den;
                ds = (rhs - sub * ds) / den;
            }
            s_sup[k * CL_X] = cp;
            s_rhs[k * CL_X] = ds;
        }
#pragma unroll 4
        for (int k = n - 2; k >= 0; --k) {
            ds = s_rhs[k * CL_X] - s_sup[k * CL_X] * ds;
            s_rhs[k * CL_X] = ds;
        }
    };
    // shear^2 (in the place of sub) and N^2 on interfaces (closure.py:150-161)
#pragma unroll 2
    for (int k = first; k <= nz; k += CL_Y) {
        real sh2 = real(0.0), nn2 = real(0.0);
        if (k >= 1 && k < nz) {
            const size_t o = (size_t)k * n2, a = o - n2;
            const real uc_prev = real(0.5) * (u[a + c] + u[a + cw]), uc = real(0.5) * (u[o + c] + u[o + cw]);
            const real vc_prev = real(0.5) * (v[a + c] + v[a + cs_]), vc = real(0.5) * (v[o + c] + v[o + cs_]);
            const real wk = wet(k), idz = g.rdzi(P, k);
            const real du = (uc_prev - uc) * idz;
            const real dv = (vc_prev - vc) * idz;
            sh2 = (du * du + dv * dv) * wk;
            // the difference of two fp64 buoyancies (their ~1e-2 relative
            // vertical contrast would lose digits in FP32)
            const real db = real((b[a + c] - b[o + c]) * idz);
            nn2 = db * wk;
        }
        s_n2[k * CL_X] = nn2;
        s_sub[k * CL_X] = sh2;
    }
    __syncthreads();
    const real depth = g.above(P, nz);
    if (P.mxl_recursive) {
        // recursive lengths (closure.py:106-129), in the place of dia: the two sweeps over
        // the column by one thread
        for (int k = first; k <= nz; k += CL_Y) {
            const real zi = g.above(P, k);
            const real zb = fmax(depth - zi, real(0.0));
            const real ek = fmax(e[(size_t)k * n2 + c], P.e_min);
            const real n2c = fmax(s_n2[k * CL_X], P.n2_min);
            const real ell = sqrt(real(2.0) * ek / n2c);
            s_dia[k * CL_X] = fmin(ell, fmin(zi + P.z_0, zb + P.z_0));
        }
        __syncthreads();
        if (threadIdx.y == 0) {
            real l = s_dia[0];
#pragma unroll 4
            for (int k = 1; k <= nz; ++k) {
                l = fmin(s_dia[k * CL_X], l + col_dzi(P, g, k));
                s_dia[k * CL_X] = l;
            }
#pragma unroll 4
            for (int k = nz - 1; k >= 0; --k) {
                l = fmin(s_dia[k * CL_X], l + col_dzi(P, g, k + 1));
                s_dia[k * CL_X] = l;
            }
        }
        __syncthreads();
    }
    // lengths and implicit TKE rows (closure.py:65-104, 171-198)
    for (int k = first; k <= nz; k += CL_Y) {
        const size_t o = (size_t)k * n2 + c;
        const real km_cur = km[o], e_old = e[o], kh_old = kh[o];
        const real km_prev = k >= 1 ? km[o - n2] : real(0.0), km_next = k < nz ? km[o + n2] : real(0.0);
        const real wk = inner(k), zi = g.above(P, k);
        const real zb = fmax(depth - zi, real(0.0));
        const real ek = fmax(e_old, P.e_min);
        // away from interface k until the energy budget is spent; once the budget is
        // zero the reference's remaining steps add exactly 0
        auto march = [&](int kk, int end, int step_k) {
            real l = real(0.0), bud = ek;
            for (; kk != end && bud > real(0.0); kk += step_k) {
                const real n2j = fmax(s_n2[kk * CL_X], real(0.0)), dzj = col_dzi(P, g, kk);
                const real cost = n2j * dzj * (l + real(0.5) * dzj);
                const bool full = cost <= bud;
                real step = dzj;
                if (!full && n2j > real(0.0)) {
                    const real part = sqrt(fmax(l * l + real(2.0) * bud / n2j, real(0.0))) - l;
                    step = fmin(fmax(part, real(0.0)), dzj);
                }
                l = l + step;
                bud = full ? bud - cost : real(0.0);
            }
            return l;
        };
        real lu, ld;
        if (!P.mxl_recursive) {
            lu = fmin(march(k - 1, -1, -1), zi + P.z_0) * wk;
            ld = fmin(march(k + 1, nz + 1, 1), zb + P.z_0) * wk;
        } else {
            lu = ld = s_dia[k * CL_X] * wk;
        }
        const real lk_k = fmax(P.l_min, sqrt(lu * ld));
        const real le_k = fmax(P.l_min, fmin(lu, ld));
        if (live) kh[o] = lk_k;  // until this thread turns it into K_h
        const real prod = (km_cur - P.nu) * s_sub[k * CL_X] - (kh_old - P.kappa) * s_n2[k * CL_X];
        const real diss = P.c_eps * sqrt(fmax(e_old, P.e_min)) / le_k;
        real a_up = real(0.0), a_dn = real(0.0);
        if (k >= 1 && k <= nz - 1) {
            const real idzi = g.rdzi(P, k);
            a_up = P.dt * (real(0.5) * (km_prev + km_cur)) * g.rdz(P, k - 1) * idzi;
            a_dn = P.dt * (real(0.5) * (km_cur + km_next)) * g.rdz(P, k) * idzi;
        }
        real sub = -a_up, sup = -a_dn;
        real diag = real(1.0) + a_up + a_dn + P.dt * diss;
        real rhs = e_old + P.dt * prod;
        if (wk <= real(0.0)) {
            diag = real(1.0);
            sub = real(0.0);
            sup = real(0.0);
            rhs = P.e_min;
        }
        if (k == 0) rhs = (g.kb > 0) ? P.e_bb * P.ustar2[c] : P.e_min;
        s_sub[k * CL_X] = sub;
        s_dia[k * CL_X] = diag;
        s_sup[k * CL_X] = sup;
        s_rhs[k * CL_X] = rhs;
    }
    __syncthreads();
    if (threadIdx.y == 0) solve(nz + 1);
    __syncthreads();
    // e/K update (closure.py:198-205)
    for (int k = first; k <= nz; k += CL_Y) {
        const size_t o = (size_t)k * n2 + c;
        const real wk = inner(k);
        real en = fmax(s_rhs[k * CL_X], P.e_min);
        en = (wk > real(0.0)) ? en : P.e_min;
        if (k == 0) en = (g.kb > 0) ? P.e_bb * P.ustar2[c] : P.e_min;
        const real kmn = P.c_k * kh[o] * sqrt(en) * wk + P.nu;
        const real kx = kmn - P.nu;
        const real khn = (P.pr_t == real(1.0) ? kx : kx / P.pr_t) + P.kappa;
        s_n2[k * CL_X] = kmn;
        if (live) {
            e[o] = en;
            km[o] = kmn;
            kh[o] = khn;
        }
    }
    __syncthreads();
    // q for the new K_m (column_q)
    for (int k = first; k < nz; k += CL_Y) {
        real sub, diag, sup;
        implicit_row_inv(P, k, g.rdz(P, k), wet(k), wet(k + 1), k == 0 ? g.rdz(P, 0) : g.rdzi(P, k),
                         k + 1 < nz ? g.rdzi(P, k + 1) : real(0.0), s_n2[k * CL_X], s_n2[(k + 1) * CL_X],
                         P.thv_dt_drag, sub, diag, sup);
        s_sub[k * CL_X] = sub;
        s_dia[k * CL_X] = diag;
        s_sup[k * CL_X] = sup;
        s_rhs[k * CL_X] = real(1.0);
    }
    __syncthreads();
    if (threadIdx.y == 0) solve(nz);
    __syncthreads();
    for (int k = first; k < nz && live; k += CL_Y) q[(size_t)k * n2 + c] = s_rhs[k * CL_X];
}

// ------------------------------------------------------------------ sums over levels
// Kernels whose levels are independent but for a running sum: a CTA takes LV_X columns
// of a row with LV_Y threads each. The threads of a column form its levels' terms
// side by side, LV_B loads deep, into shared memory; then one warp per sum adds them
// in the order of the levels. With a thread per column (32 x 4 a CTA) a level waits for
// the one before it, and a 128 x 128 grid puts one warp on each scheduler.
constexpr int LV_X = 32, LV_Y = 8, LV_B = 4, LV_K = LV_Y * LV_B;

// Columns up to which a thread per column leaves the SMs short of warps. Above, the
// column's geometry, which every thread of it works out again, costs more than the
// waiting. us a launch by columns and by levels: w at 16,384 x 50 64 and 23, at 46,937 x 37
// 48 and 41, at 122,880 x 30 54 and 86, at 262,144 x 50 198 and 330; the back substitution at
// 16,384 x 50 29 and 8, at 46,937 x 37 27 and 14, at 262,144 x 50 82 and 88; Ku and Kv (three
// columns' geometry for little arithmetic: half the limit) at 16,384 x 50 35 and 13, at
// 46,937 x 37 22 and 26. One grid alone still gains at 65,536 (back substitution 26 and 16),
// but eight members of an ensemble, which fill the GPU together, lost 5% there.
// Each kernel has less to gain where a column has few levels, and those that keep a
// column's rows in shared memory where it has many: their limits below, from both forms
// timed at 4,096 to 49,152 columns of 4 to 128 levels.
constexpr int kFewColumns = 49152;
constexpr bool kFp64 = sizeof(real) == 8;

// Sums over levels (w, Ku and Kv): a chunk costs LV_K levels however many it has. us a launch of
// w by columns and by levels: 43,264 x 64 82 and 61, x 24 33 and 31, x 16 24 and 29, x 8 16 and
// 25; 33,792 x 16 24 and 22, x 8 16 and 21; 25,600 x 8 15 and 19; 20,448 x 12 within 2%; of two
// chunks 43,264 x 40 within 2%, x 33 43 and 47, 46,937 x 37 48 and 41.
static int level_sum_columns(int nz) {
    const int slots = (nz + LV_K - 1) / LV_K * LV_K;
    if (2 * nz < slots) return 98304 * nz / slots - 16384;
    return 100 * nz < (nz <= LV_K ? 60 : 55) * slots ? 36864 : kFewColumns;
}

// Back substitution: with fewer levels than a column has threads, and in FP32 up to two levels
// a thread, the columns' form is as fast or faster from there on (us by columns and by levels:
// 33,792 x 4 10.9 and 12.1, 23,040 x 4 11.1 and 10.3; FP32 49,152 x 8 10.0 and 11.0, 33,792 x 12 11.0
// and 10.6).
static int backsub_columns(int nz) {
    if (nz < LV_Y) return kFp64 ? 24576 : 16384;
    return !kFp64 && nz < 2 * LV_Y ? 36864 : kFewColumns;
}

// CTAs with that much dynamic shared memory that an SM holds: of its 228 KB a CTA takes 1 KB
// more than it asks for
static int smem_ctas(size_t bytes) { return (int)((228 * 1024) / (bytes + 1024)); }

// Closure: with one CTA an SM (from 90 levels on in fp64) from about 27,000 columns on the
// columns' form is faster (us by columns and by levels: 43,264 x 88 592 and 425, x 104 719
// and 907; 25,600 x 104 634 and 527), and with few levels, where the lengths' marches are short,
// earlier too (43,264 x 8 42 and 51, 25,600 x 8 37 and 30; FP32 43,264 x 8 29 and 29).
static int closure_columns(int nz) {
    const int limit = smem_ctas((size_t)5 * (nz + 1) * 32 * sizeof(real)) >= 2 ? kFewColumns : 26624;
    const int shallow = (kFp64 ? 21504 : 32768) + 1024 * nz;
    return nz < (kFp64 ? 14 : 10) && shallow < limit ? shallow : limit;
}

// Tracer solve: the two eliminations stay with one warp in four, so the lines lie lower.
// us by columns and by levels: 43,264 x 128 285 and 475, x 88 199 and 195, x 64 143 and 146, x 40
// 86 and 78, x 24 47 and 52, x 8 20 and 25; 25,600 x 104 200 and 230, x 24 41 and 33; FP32 43,264 x
// 128 238 and 206, x 24 38 and 37, x 16 28 and 28, x 8 17 and 19.
static int tracer_columns(int nz) {
    if (nz < 8) return 16384;
    if (!kFp64) return nz < 20 ? 36864 : kFewColumns;
    if (nz < 32) return nz < 24 ? 25600 : 28672;
    const int ctas = smem_ctas((size_t)5 * nz * 32 * sizeof(real));
    return ctas >= 3 ? kFewColumns : ctas == 2 ? 40960 : 16384;
}

#define LEVELS_PROLOGUE                                          \
    const int lv_tiles = (P.nx + LV_X - 1) / LV_X;               \
    const int j = blockIdx.x / lv_tiles;                         \
    const int lv_i = (blockIdx.x - j * lv_tiles) * LV_X + threadIdx.x; \
    const bool live = lv_i < P.nx; /* the others repeat the last column and store nothing */ \
    const int i = live ? lv_i : P.nx - 1;                        \
    Nbr nb;                                                      \
    nb.init(i, j, P.nx, P.ny);                                   \
    const size_t n2 = (size_t)P.n2;                              \
    (void)n2;                                                    \
    (void)live;

template <class T>
static dim3 level_grid(const KPT<T>& P) { return dim3((unsigned)(((P.nx + LV_X - 1) / LV_X) * P.ny)); }
static dim3 level_block() { return dim3(LV_X, LV_Y); }

// NS running sums over the levels 0 .. nz - 1 (UP: nz - 1 .. 0): term(k, t) forms level k's
// terms t[NS]; after each chunk of LV_K levels warp n < NS adds its sum's, calling
// step(n, k, sum) after each level. sum starts with the first level's term.
template <int NS, bool UP, class T, class F, class G>
__device__ __forceinline__ void level_sums(int nz, T (*terms)[LV_K][LV_X], F term, G step) {
    T sum = T(0.0);
    for (int c0 = 0; c0 < nz; c0 += LV_K) {
        const int n = nz - c0 < LV_K ? nz - c0 : LV_K;
#pragma unroll
        for (int q = 0; q < LV_B; ++q) {
            const int r = threadIdx.y + q * LV_Y, rc = r < n ? r : n - 1;
            T t[NS];
            term(UP ? nz - 1 - (c0 + rc) : c0 + rc, t);
#pragma unroll
            for (int m = 0; m < NS; ++m) terms[m][r][threadIdx.x] = t[m];
        }
        __syncthreads();
        if (threadIdx.y < NS) {
#pragma unroll 4
            for (int r = 0; r < n; ++r) {
                const T t = terms[threadIdx.y][r][threadIdx.x];
                sum = (c0 + r == 0) ? t : sum + t;
                step(threadIdx.y, UP ? nz - 1 - (c0 + r) : c0 + r, sum);
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------ Ku, Kv
// Ku = sum_k dz3u * min(q, q_east) * mask_u (model3d_v05.py:154-157)
__global__ void k_kukv(KPR P, const real* __restrict__ q, wide* __restrict__ Ku,
                       wide* __restrict__ Kv) {
    COLUMN_PROLOGUE
    const size_t c = nb.c;
    const size_t ce = nb.at(0, 1), cn = nb.at(1, 0);
    const ColGeoR gc = ColGeoR::load(P, (int)c), ge = ColGeoR::load(P, (int)ce), gn = ColGeoR::load(P, (int)cn);
    const int2 kf = P.kface[c];
    wide su = 0.0, sv = 0.0;  // depth sums in fp64 on both paths
#pragma unroll 4
    for (int k = 0; k < P.nz; ++k) {
        const size_t o = (size_t)k * n2;
        real m;
        const real dzc = gc.dz(P, k, m), dze = ge.dz(P, k, m), dzn = gn.dz(P, k, m);
        const real qc = q[o + c];
        const real tu = face_dz(P, kf.x, k, dzc, dze) * fmin(qc, q[o + ce]);
        const real tv = face_dz(P, kf.y, k, dzc, dzn) * fmin(qc, q[o + cn]);
        su = (k == 0) ? wide(tu) : su + wide(tu);
        sv = (k == 0) ? wide(tv) : sv + wide(tv);
    }
    Ku[c] = su * P.mask_u64[c];
    Kv[c] = sv * P.mask_v64[c];
}

// the same by levels, for few columns
__global__ void __launch_bounds__(LV_X * LV_Y, 4) k_kukv_few(KPR P, const real* __restrict__ q, wide* __restrict__ Ku,
                                                      wide* __restrict__ Kv) {
    __shared__ wide terms[2][LV_K][LV_X];
    LEVELS_PROLOGUE
    const size_t c = nb.c;
    const size_t ce = nb.at(0, 1), cn = nb.at(1, 0);
    const ColGeoR gc = ColGeoR::load(P, (int)c), ge = ColGeoR::load(P, (int)ce), gn = ColGeoR::load(P, (int)cn);
    const int2 kf = P.kface[c];
    const int nz = P.nz;
    // depth sums in fp64 on both paths
    level_sums<2, false>(nz, terms, [&](int k, wide* t) {
        const size_t o = (size_t)k * n2;
        real m;
        const real dzc = gc.dz(P, k, m), dze = ge.dz(P, k, m), dzn = gn.dz(P, k, m);
        const real qc = q[o + c];
        t[0] = wide(face_dz(P, kf.x, k, dzc, dze) * fmin(qc, q[o + ce]));
        t[1] = wide(face_dz(P, kf.y, k, dzc, dzn) * fmin(qc, q[o + cn]));
    }, [&](int n, int k, wide sum) {
        if (k == nz - 1 && live) (n ? Kv : Ku)[c] = sum * (n ? P.mask_v64 : P.mask_u64)[c];
    });
}

// ------------------------------------------------------------------ w from transport divergence
// w[k] = -sum_{k'>=k} div(dz3u u, dz3v v)[k'], accumulated from the bottom
// (vertical_var.py:109-121); w[nz] = 0.
__global__ void __launch_bounds__(128, 8) k_wcol(KPR P, const real* __restrict__ u, const real* __restrict__ v,
                       real* __restrict__ w) {
    COLUMN_PROLOGUE
    const int nz = P.nz;
    const size_t c = nb.c, cw = nb.at(0, -1), cs_ = nb.at(-1, 0);
    const ColGeoR gc = ColGeoR::load(P, (int)c), ge = ColGeoR::load(P, nb.at(0, 1)),
                 gw = ColGeoR::load(P, (int)cw), gn = ColGeoR::load(P, nb.at(1, 0)), gs = ColGeoR::load(P, (int)cs_);
    const int2 kf = P.kface[c];
    const int kuw = P.kface[cw].x, kvs = P.kface[cs_].y;
    real acc = real(0.0);
    w[(size_t)nz * n2 + c] = real(0.0);
#pragma unroll 2
    for (int k = nz - 1; k >= 0; --k) {
        const size_t o = (size_t)k * n2;
        real m3, m;
        const real dzc = gc.dz(P, k, m3);
        const real dzu_c = face_dz(P, kf.x, k, dzc, ge.dz(P, k, m));
        const real dzu_w = face_dz(P, kuw, k, gw.dz(P, k, m), dzc);
        const real dzv_c = face_dz(P, kf.y, k, dzc, gn.dz(P, k, m));
        const real dzv_s = face_dz(P, kvs, k, gs.dz(P, k, m), dzc);
        const real td = m3 * ((dzu_c * u[o + c] - dzu_w * u[o + cw]) / P.dx +
                                (dzv_c * v[o + c] - dzv_s * v[o + cs_]) / P.dy);
        acc = (k == nz - 1) ? td : acc + td;
        w[o + c] = -acc;
    }
}

// the same by levels, for few columns
__global__ void __launch_bounds__(LV_X * LV_Y, 4) k_wcol_few(KPR P, const real* __restrict__ u, const real* __restrict__ v,
                                                      real* __restrict__ w) {
    __shared__ real terms[1][LV_K][LV_X];
    LEVELS_PROLOGUE
    const int nz = P.nz;
    const size_t c = nb.c, cw = nb.at(0, -1), cs_ = nb.at(-1, 0);
    const ColGeoR gc = ColGeoR::load(P, (int)c), ge = ColGeoR::load(P, nb.at(0, 1)),
                 gw = ColGeoR::load(P, (int)cw), gn = ColGeoR::load(P, nb.at(1, 0)), gs = ColGeoR::load(P, (int)cs_);
    const int2 kf = P.kface[c];
    const int kuw = P.kface[cw].x, kvs = P.kface[cs_].y;
    if (threadIdx.y == 0 && live) w[(size_t)nz * n2 + c] = real(0.0);
    level_sums<1, true>(nz, terms, [&](int k, real* t) {
        const size_t o = (size_t)k * n2;
        real m3, m;
        const real dzc = gc.dz(P, k, m3);
        const real dzu_c = face_dz(P, kf.x, k, dzc, ge.dz(P, k, m));
        const real dzu_w = face_dz(P, kuw, k, gw.dz(P, k, m), dzc);
        const real dzv_c = face_dz(P, kf.y, k, dzc, gn.dz(P, k, m));
        const real dzv_s = face_dz(P, kvs, k, gs.dz(P, k, m), dzc);
        t[0] = m3 * ((dzu_c * u[o + c] - dzu_w * u[o + cw]) / P.dx + (dzv_c * v[o + c] - dzv_s * v[o + cs_]) / P.dy);
    }, [&](int, int k, real sum) {
        if (live) w[(size_t)k * n2 + c] = -sum;
    });
}

// ------------------------------------------------------------------ buoyancy potential
// phi[k] = 0.5 dz3 b + sum_{k'<k} dz3 b, optionally minus its thickness-weighted
// column mean (vertical_var.py:132-145).
__global__ void k_phi(KPR P, const wide* __restrict__ b, wide* __restrict__ phi) {
    // fp64 on both paths: neighbouring columns' potentials of ~1e3 m2 s-2 differ
    // by the baroclinic pressure signal, which FP32 would not resolve
    COLUMN_PROLOGUE
    const int nz = P.nz;
    const size_t c = nb.c;
    const ColGeo64 g = ColGeo64::load(P, (int)c);
    wide above = 0.0, total = 0.0;
#pragma unroll 4
    for (int k = 0; k < nz; ++k) {
        const size_t o = (size_t)k * n2 + c;
        const wide dz = g.dz(P, k);
        const wide bk = b[o];
        phi[o] = 0.5 * dz * bk + above;
        const wide t = dz * bk;
        above = (k == 0) ? t : above + t;
        total = (k == 0) ? dz : total + dz;
    }
    if (P.pgf_remove) {
        wide s = 0.0;
        for (int k = 0; k < nz; ++k) {
            const wide dz = g.dz(P, k);
            const wide t = dz * phi[(size_t)k * n2 + c];
            s = (k == 0) ? t : s + t;
        }
        const wide mean = s * inv_pos(total);
        for (int k = 0; k < nz; ++k) {
            const size_t o = (size_t)k * n2 + c;
            phi[o] = phi[o] - mean;
        }
    }
}

// ------------------------------------------------------------------ stencil accessors
// The horizontal stencils below read the face velocities and face masks of one
// level through an accessor: U(dj, di) / V(dj, di) are u / v of column
// (j + dj, i + di), MU / MV the 0/1 wet flags of its east / north face.
struct GlobalLevel {  // straight from the level planes in global memory
    const KPR& P;
    const Nbr& nb;
    const real* __restrict__ u;
    const real* __restrict__ v;
    size_t o;
    int k;
    __device__ __forceinline__ real U(int dj, int di) const { return u[o + nb.at(dj, di)]; }
    __device__ __forceinline__ real V(int dj, int di) const { return v[o + nb.at(dj, di)]; }
    __device__ __forceinline__ real MU(int dj, int di) const { return col_m3u(P, nb.at(dj, di), k); }
    __device__ __forceinline__ real MV(int dj, int di) const { return col_m3v(P, nb.at(dj, di), k); }
};

// ------------------------------------------------------------------ Coriolis averages
// v averaged onto u points over wet v faces (operators_masked.py:45-52)
template <class A>
__device__ __forceinline__ real v_on_u_at(const A& a) {
    const real f0 = a.V(0, 0), f1 = a.V(-1, 0), f2 = a.V(0, 1), f3 = a.V(-1, 1);
    const real w0 = a.MV(0, 0), w1 = a.MV(-1, 0), w2 = a.MV(0, 1), w3 = a.MV(-1, 1);
    real num = real(0.0) + w0 * f0;
    num = num + w1 * f1;
    num = num + w2 * f2;
    num = num + w3 * f3;
    real den = real(0.0) + w0;
    den = den + w1;
    den = den + w2;
    den = den + w3;
    const real avg = den > real(0.0) ? num / den : real(0.0);
    return avg * a.MU(0, 0);
}

// u averaged onto v points over wet u faces (operators_masked.py:55-61)
template <class A>
__device__ __forceinline__ real u_on_v_at(const A& a) {
    const real f0 = a.U(0, 0), f1 = a.U(0, -1), f2 = a.U(1, 0), f3 = a.U(1, -1);
    const real w0 = a.MU(0, 0), w1 = a.MU(0, -1), w2 = a.MU(1, 0), w3 = a.MU(1, -1);
    real num = real(0.0) + w0 * f0;
    num = num + w1 * f1;
    num = num + w2 * f2;
    num = num + w3 * f3;
    real den = real(0.0) + w0;
    den = den + w1;
    den = den + w2;
    den = den + w3;
    const real avg = den > real(0.0) ? num / den : real(0.0);
    return avg * a.MV(0, 0);
}

__device__ __forceinline__ real v_on_u(const KPR& P, const Nbr& nb, const real* __restrict__ v, size_t o,
                                         int k) {
    return v_on_u_at(GlobalLevel{P, nb, nullptr, v, o, k});
}

__device__ __forceinline__ real u_on_v(const KPR& P, const Nbr& nb, const real* __restrict__ u, size_t o,
                                         int k) {
    return u_on_v_at(GlobalLevel{P, nb, u, nullptr, o, k});
}

// horizontal Laplacian D o G with the given face masks (operators_masked.py:64-68);
// which = 0: u (x-mask m3u, y-mask m3v, cell mask m3u), 1: v (cell mask m3v),
// 2: tracer (cell mask m3)
__device__ real hlap(const KPR& P, const Nbr& nb, const real* __restrict__ f, int k, int which) {
    const size_t o = (size_t)k * P.n2;
    auto F = [&](int dj, int di) { return f[o + nb.at(dj, di)]; };
    const real gx0 = m3u_at(P, nb, 0, 0, k) * (F(0, 1) - F(0, 0)) / P.dx;
    const real gxw = m3u_at(P, nb, 0, -1, k) * (F(0, 0) - F(0, -1)) / P.dx;
    const real gy0 = m3v_at(P, nb, 0, 0, k) * (F(1, 0) - F(0, 0)) / P.dy;
    const real gys = m3v_at(P, nb, -1, 0, k) * (F(0, 0) - F(-1, 0)) / P.dy;
    const real m = which == 0 ? m3u_at(P, nb, 0, 0, k)
                                : (which == 1 ? m3v_at(P, nb, 0, 0, k) : m3_at(P, nb, 0, 0, k));
    return m * ((gx0 - gxw) / P.dx + (gy0 - gys) / P.dy);
}

// explicit vertical diffusion of a face velocity (vertical_var.py:80-106) with
// the column's interface viscosity, the face thickness table dzf[k-1..k+1], the
// cell mask's bottom rule and surface flux `surf`
__device__ __forceinline__ real explicit_dz(const KPR& P, int k, real fkm1, real fk, real fkp1,
                                              real Kk, real Kk1, real dzf_m1, real dzf_k,
                                              real dzf_p1, real m3k_m1_bottom,
                                              real m3k_bottom, real m3k, real surf,
                                              real drag) {
    const int nz = P.nz;
    real flux_k, flux_k1;
    if (k == 0) {
        flux_k = surf;
    } else {
        const real dzi = real(0.5) * (dzf_m1 + dzf_k);
        flux_k = Kk * (fkm1 - fk) * inv_pos(dzi);
        if (m3k_m1_bottom > real(0.0)) flux_k = real(0.0);
    }
    if (k == nz - 1) {
        flux_k1 = real(0.0);
    } else {
        const real dzi = real(0.5) * (dzf_k + dzf_p1);
        flux_k1 = Kk1 * (fk - fkp1) * inv_pos(dzi);
        if (m3k_bottom > real(0.0)) flux_k1 = real(0.0);
    }
    const real idz = inv_pos(dzf_k);
    const real out = (flux_k - flux_k1) * idz;
    const real dragc = drag * fk * m3k_bottom;
    return (out - dragc * idz) * (m3k > real(0.0) ? real(1.0) : real(0.0));
}

// ------------------------------------------------------------------ momentum advection
// x- and y-flux divergence of u at its east face (advection_v06.py:77-99 for the
// kappa/TVD scheme, advection.py:62-79 for the centred one); the reference forms
// ax + ay + az left to right, so (ax + ay) + az is its sum
template <class A>
__device__ __forceinline__ real mom_adv_u_xy(const KPR& P, const A& a) {
    if (P.advection >= 3) {
        const bool lim = P.advection == 4;
        const real ub_c0 = real(0.5) * (a.U(0, -1) + a.U(0, 0));
        const real ub_c1 = real(0.5) * (a.U(0, 0) + a.U(0, 1));
        const real uc0 = kappa_face(P, a.U(0, -2), a.U(0, -1), a.U(0, 0), a.U(0, 1), ub_c0, a.MU(0, -2),
                                      a.MU(0, 1), lim);
        const real uc1 = kappa_face(P, a.U(0, -1), a.U(0, 0), a.U(0, 1), a.U(0, 2), ub_c1, a.MU(0, -1),
                                      a.MU(0, 2), lim);
        const real ax = (ub_c1 * uc1 - ub_c0 * uc0) / P.dx;
        const real vb0 = real(0.5) * (a.V(0, 0) + a.V(0, 1));
        const real vbm = real(0.5) * (a.V(-1, 0) + a.V(-1, 1));
        const real fy0 = vb0 * kappa_face(P, a.U(-1, 0), a.U(0, 0), a.U(1, 0), a.U(2, 0), vb0, a.MU(-1, 0),
                                            a.MU(2, 0), lim);
        const real fym = vbm * kappa_face(P, a.U(-2, 0), a.U(-1, 0), a.U(0, 0), a.U(1, 0), vbm, a.MU(-2, 0),
                                            a.MU(1, 0), lim);
        return ax + (fy0 - fym) / P.dy;
    }
    const real ub_c0 = real(0.5) * (a.U(0, -1) + a.U(0, 0));
    const real ub_c1 = real(0.5) * (a.U(0, 0) + a.U(0, 1));
    const real ax = (ub_c1 * ub_c1 - ub_c0 * ub_c0) / P.dx;
    const real vb0 = real(0.5) * (a.V(0, 0) + a.V(0, 1));
    const real vbm = real(0.5) * (a.V(-1, 0) + a.V(-1, 1));
    const real fy0 = vb0 * (real(0.5) * (a.U(0, 0) + a.U(1, 0)));
    const real fym = vbm * (real(0.5) * (a.U(-1, 0) + a.U(0, 0)));
    return ax + (fy0 - fym) / P.dy;
}

// the same for v at its north face (advection_v06.py:100-108, advection.py:81-95):
// bx + by, formed in that order
template <class A>
__device__ __forceinline__ real mom_adv_v_xy(const KPR& P, const A& a) {
    if (P.advection >= 3) {
        const bool lim = P.advection == 4;
        const real vb_c0 = real(0.5) * (a.V(-1, 0) + a.V(0, 0));
        const real vb_c1 = real(0.5) * (a.V(0, 0) + a.V(1, 0));
        const real vc0 = kappa_face(P, a.V(-2, 0), a.V(-1, 0), a.V(0, 0), a.V(1, 0), vb_c0, a.MV(-2, 0),
                                      a.MV(1, 0), lim);
        const real vc1 = kappa_face(P, a.V(-1, 0), a.V(0, 0), a.V(1, 0), a.V(2, 0), vb_c1, a.MV(-1, 0),
                                      a.MV(2, 0), lim);
        const real by = (vb_c1 * vc1 - vb_c0 * vc0) / P.dy;
        const real ub0 = real(0.5) * (a.U(0, 0) + a.U(1, 0));
        const real ubm = real(0.5) * (a.U(0, -1) + a.U(1, -1));
        const real fx0 = ub0 * kappa_face(P, a.V(0, -1), a.V(0, 0), a.V(0, 1), a.V(0, 2), ub0, a.MV(0, -1),
                                            a.MV(0, 2), lim);
        const real fxm = ubm * kappa_face(P, a.V(0, -2), a.V(0, -1), a.V(0, 0), a.V(0, 1), ubm, a.MV(0, -2),
                                            a.MV(0, 1), lim);
        return (fx0 - fxm) / P.dx + by;
    }
    const real vb_c0 = real(0.5) * (a.V(-1, 0) + a.V(0, 0));
    const real vb_c1 = real(0.5) * (a.V(0, 0) + a.V(1, 0));
    const real by = (vb_c1 * vb_c1 - vb_c0 * vb_c0) / P.dy;
    const real ub0 = real(0.5) * (a.U(0, 0) + a.U(1, 0));
    const real ubm = real(0.5) * (a.U(0, -1) + a.U(1, -1));
    const real fx0 = ub0 * (real(0.5) * (a.V(0, 0) + a.V(0, 1)));
    const real fxm = ubm * (real(0.5) * (a.V(0, -1) + a.V(0, 0)));
    return (fx0 - fxm) / P.dx + by;
}

// advective flux of a face velocity through interface kk of its column (0 =
// surface), from the velocity at kk-2 .. kk+1, the interface w averaged over
// the two cells of the face, and the face's wet levels kf
// (advection_v06.py:50-74 and :86-99; advection.py:75-79)
__device__ __forceinline__ real mom_vflux(const KPR& P, int kk, int kf, real f_m2, real f_m1, real f_0,
                                            real f_p1, real wa, real wb_) {
    const int nz = P.nz;
    if (kk == 0 || kk == nz) return real(0.0);
    const real wb = real(0.5) * (wa + wb_);
    if (P.advection >= 3) {
        const real fu = (kk >= 2) ? f_m2 : real(0.0);
        const real fd = (kk + 1 <= nz - 1) ? f_p1 : real(0.0);
        const bool hu = (kk >= 2) && kk - 2 < kf;
        const bool hd = (kk + 1 <= nz - 1) && kk + 1 < kf;
        return wb * kappa_face_z(P, fu, f_m1, f_0, fd, wb, hu, hd, P.advection == 4);
    }
    return wb * real(0.5) * (f_m1 + f_0);
}

// the diffusive flux K (f_above - f_below) / dzi through interface k of a face
// velocity column (vertical_var.py:80-106), zero when the level above is the
// column's last wet one
__device__ __forceinline__ real diff_flux(real Kk, real f_above, real f_below, real dzf_above,
                                           real dzf_below, real bottom_above) {
    const real dzi = real(0.5) * (dzf_above + dzf_below);
    const real flux = Kk * (f_above - f_below) * inv_pos(dzi);
    return bottom_above > real(0.0) ? real(0.0) : flux;
}

// ------------------------------------------------------------------ explicit momentum terms
// Everything of the predictor that depends on the old state only: the
// common-depth pressure gradient, the old-state Coriolis average, the explicit
// vertical diffusion and the stress + advection/viscosity increment
// (model3d_v05.py:352-370), in level-marching form: two threads per column of
// a 32 x 8 tile, one for the u terms and one for the v terms, march P.mom_kl
// levels over the level planes the CTA stages in shared memory. The compact
// geometry of the column and of its face's far neighbour is formed once; the
// component's velocity and face thickness at the levels above and below roll
// in registers; the vertical advective flux at the bottom of a level and the
// diffusive flux there are carried to the next level as the fluxes at its top
// (a per-cell form forms each of them twice). Every value is formed by the
// reference's operations in its order.
constexpr int MOM_TX = 32, MOM_TY = 8, MOM_RX = MOM_TX + 4, MOM_RY = MOM_TY + 4, MOM_RN = MOM_RX * MOM_RY;

// The right-hand side of a momentum tridiagonal at one cell: the explicit predictor with
// the Coriolis average `av` of the old state and `it` of the iterate, plus the
// stress/advection increment (model3d_v05.py:387-393); f is f0 for u, -f0 for v.
__device__ __forceinline__ real predictor(const KPR& P, real x, real f, real av, real it, real pg, real g2, real m,
                                          real dz, real st) {
    const real cor = P.one_m_tc * av + P.theta_cor * it;
    real g = x + P.dt * (f * cor + pg);
    if (P.scheme != 2) g = g - P.c1 * (g2 * m);
    g = g + P.c3 * dz;
    return g + st;
}

// the level's u, v and face masks of a tile plus a 2-column ring, in shared memory
struct TileLevel {
    const real* su;
    const real* sv;
    const int* sku;
    const int* skv;
    int rc;  // the thread's column in the region
    int k;
    __device__ __forceinline__ real U(int dj, int di) const { return su[rc + dj * MOM_RX + di]; }
    __device__ __forceinline__ real V(int dj, int di) const { return sv[rc + dj * MOM_RX + di]; }
    __device__ __forceinline__ real MU(int dj, int di) const { return k < sku[rc + dj * MOM_RX + di] ? real(1.0) : real(0.0); }
    __device__ __forceinline__ real MV(int dj, int di) const { return k < skv[rc + dj * MOM_RX + di] ? real(1.0) : real(0.0); }
};

// What a level does to the values carried down a face's column.
struct MomCarry {
    real x_m1, x_0, x_p1;  // the component's velocity at levels k - 1, k, k + 1
    real fz, df;           // vertical advective and diffusive flux through the top of level k
};

// The outputs of one component, by pointer (its own arrays of the eight, plus the right-hand side)
struct MomOut {
    real *pg, *av, *dz, *st, *rhs;
};

// One level of a tile whose columns, ring included, are wet and full at levels k and
// k + 1: thicknesses and their reciprocals come from the level table, the two columns
// of a face sit at one depth, and the face masks are those of the 2D faces (fl: bit per
// stencil place, see mom_face_flags). COMP 0 is u: `along` is x and the other velocity
// v; COMP 1 is v: along y, u. The terms are those of the general form below, operation
// for operation; where a factor is 1 or a difference of equal depths 0 it is left out.
template <int COMP>
__device__ __forceinline__ void mom_full_level(const KLR& P, const real* __restrict__ X, const real* __restrict__ Y,
                                               unsigned fl, int kff, int k, real x_p2, real K_1, real w_c, real w_f,
                                               wide phc, wide phf, wide bc, wide bf, real tau, real g2, size_t at,
                                               const MomOut& out, MomCarry& q) {
    constexpr int A = COMP ? MOM_RX : 1, B = COMP ? 1 : MOM_RX;  // strides along the component's axis and across it
    const real m = (fl >> 8) & 1 ? real(1.0) : real(0.0);
    const wide dxy = COMP ? P.dy64 : P.dx64;
    wide pgw;
    if (P.pgf_correction) pgw = m * ((phf + bf * 0.0) - (phc + bc * 0.0)) / dxy;
    else pgw = m * (phf - phc) / dxy * m;
    const real pg = real(pgw);
    out.pg[at] = pg;
    // Coriolis average over the wet ones of four faces
    const real y0 = Y[0], y1 = Y[-B], y2 = Y[A], y3 = Y[A - B];
    real av;
    if ((fl >> 9 & 15u) == 15u) {
        av = (((y0 + y1) + y2) + y3) * real(0.25) * m;  // a division by 4 is exact
    } else {
        const real w0 = (fl >> 9) & 1, w1 = (fl >> 10) & 1, w2 = (fl >> 11) & 1, w3 = (fl >> 12) & 1;
        const real den = ((w0 + w1) + w2) + w3;
        const real num = ((w0 * y0 + w1 * y1) + w2 * y2) + w3 * y3;
        av = (den > real(0.0) ? num / den : real(0.0)) * m;
    }
    out.av[at] = av;
    // explicit vertical diffusion
    const bool open = (fl >> 8) & 1;  // a closed face has no thickness
    const real db = K_1 * (q.x_0 - q.x_p1) * (open ? P.rfdzi[k + 1] : real(0.0));
    const real rdz = open ? P.rfdz[k] : real(0.0);
    const real dz = (q.df - db) * rdz;
    out.dz[at] = dz;
    // advection
    real ex = real(0.0), fb = real(0.0);
    const real xa1 = X[-A], x0 = X[0], xb1 = X[A], xc1 = X[-B], xd1 = X[B];
    if (P.advection != 0) {
        fb = mom_vflux(P, k + 1, kff, q.x_m1, q.x_0, q.x_p1, x_p2, w_c, w_f);
        const real a0 = real(0.5) * (xa1 + x0), a1 = real(0.5) * (x0 + xb1);      // along, at the cell centres
        const real b0 = real(0.5) * (y0 + y2), bm = real(0.5) * (y1 + y3);        // across, at the corners
        real al, ac;
        if (P.advection >= 3) {
            const bool lim = P.advection == 4;
            const real c0 = kappa_face_f(P, X[-2 * A], xa1, x0, xb1, a0, fl & 1, fl & 2, lim);
            const real c1 = kappa_face_f(P, xa1, x0, xb1, X[2 * A], a1, fl & 4, fl & 8, lim);
            al = a1 * c1 - a0 * c0;
            const real f0 = b0 * kappa_face_f(P, xc1, x0, xd1, X[2 * B], b0, fl & 16, fl & 32, lim);
            const real fm = bm * kappa_face_f(P, X[-2 * B], xc1, x0, xd1, bm, fl & 64, fl & 128, lim);
            ac = f0 - fm;
        } else {
            al = a1 * a1 - a0 * a0;
            const real f0 = b0 * (real(0.5) * (x0 + xd1));
            const real fm = bm * (real(0.5) * (xc1 + x0));
            ac = f0 - fm;
        }
        const real h = COMP ? ac / P.dx + al / P.dy : al / P.dx + ac / P.dy;
        const real a = h + (q.fz - fb) / P.dz_nom[k];
        ex = ex - a * m;
    }
    if (P.a_h > real(0.0)) {
        // horizontal Laplacian with face masks (hlap): of the cells around u, the x faces
        // carry the u masks and the y faces the v masks; the same around v
        const real g0 = ((fl >> (COMP ? 9 : 8)) & 1 ? real(1.0) : real(0.0)) * ((COMP ? xd1 : xb1) - x0) / P.dx;
        const real gw = ((fl >> (COMP ? 10 : 2)) & 1 ? real(1.0) : real(0.0)) * (x0 - (COMP ? xc1 : xa1)) / P.dx;
        const real h0 = ((fl >> (COMP ? 8 : 9)) & 1 ? real(1.0) : real(0.0)) * ((COMP ? xb1 : xd1) - x0) / P.dy;
        const real hs = ((fl >> (COMP ? 2 : 10)) & 1 ? real(1.0) : real(0.0)) * (x0 - (COMP ? xa1 : xc1)) / P.dy;
        ex = ex + P.a_h * (m * ((g0 - gw) / P.dx + (h0 - hs) / P.dy));
    }
    const real st = (k == 0) ? P.thv_dt * tau * rdz + P.dt * ex : real(0.0) + P.dt * ex;
    out.st[at] = st;
    out.rhs[at] = predictor(P, x0, COMP ? P.neg_f0 : P.f0, av, av, pg, g2, m, dz, st);
    q.fz = fb;
    q.df = db;
    q.x_m1 = q.x_0;
    q.x_0 = q.x_p1;
    q.x_p1 = x_p2;
}

// the open faces of a component's stencil (region column rc; A, B: strides along its
// axis and across; own and oth: wet levels of the faces of this and the other
// component), one bit each: far cells of the two faces along (0..3) and across (4..7),
// the face itself (8), the four faces of the Coriolis average (9..12)
__device__ __forceinline__ unsigned mom_face_flags(const int* own, const int* oth, int rc, int A, int B) {
    unsigned f = 0;
    f |= (own[rc - 2 * A] > 0) << 0 | (own[rc + A] > 0) << 1 | (own[rc - A] > 0) << 2 | (own[rc + 2 * A] > 0) << 3;
    f |= (own[rc - B] > 0) << 4 | (own[rc + 2 * B] > 0) << 5 | (own[rc - 2 * B] > 0) << 6 | (own[rc + B] > 0) << 7;
    f |= (own[rc] > 0) << 8;
    f |= (oth[rc] > 0) << 9 | (oth[rc - B] > 0) << 10 | (oth[rc + A] > 0) << 11 | (oth[rc + A - B] > 0) << 12;
    return f;
}

// Bound by instruction issue, most of it the limiter's selects and divisions (five per
// component and level that depend on data). Over a flat or gently sloping bottom most
// levels of a tile are wet and full in every column, ring included, so a CTA first marches
// those (mom_full_level) -- no thickness, depth or mask of any column is formed there
// -- and the levels below in the general form. The first pass's right-hand sides are formed
// here too, from values in registers: a pass over twelve arrays less. us a launch at
// 512 x 512 x 50: 1114 before with 242 of a first k_predictor_rhs beside it, 1043 now (FP32 751
// with 159, now 636).
__global__ void __launch_bounds__(MOM_TX * MOM_TY * 2, OC_MINB_MOM) k_mom_column(
    KLR P, const real* __restrict__ u, const real* __restrict__ v, const wide* __restrict__ b,
    const wide* __restrict__ phi, const real* __restrict__ w, const real* __restrict__ km,
    const wide* __restrict__ gx2, const wide* __restrict__ gy2, real* __restrict__ pgx, real* __restrict__ pgy,
    real* __restrict__ avpv, real* __restrict__ avpu, real* __restrict__ dzu, real* __restrict__ dzv,
    real* __restrict__ stu, real* __restrict__ stv, real* __restrict__ ru, real* __restrict__ rv) {
    __shared__ int s_ku[MOM_RN], s_kv[MOM_RN];
    __shared__ int s_full;
    __shared__ real s_u[2][MOM_RN], s_v[2][MOM_RN];  // level planes, double-buffered
    // threadIdx.z selects the component: 0 the u terms at the column's east face,
    // 1 the v terms at its north face (whole warps, so no divergence)
    const int tx = threadIdx.x, ty = threadIdx.y, comp = threadIdx.z;
    const int tid = (comp * MOM_TY + ty) * MOM_TX + tx;
    constexpr int NT = MOM_TX * MOM_TY * 2, NS = (MOM_RN + NT - 1) / NT;  // threads, region columns per thread
    const int i0 = blockIdx.x * MOM_TX, j0 = blockIdx.y * MOM_TY;
    const int i = i0 + tx, j = j0 + ty;
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    const bool live = i < nx && j < ny;
    const int kbeg = blockIdx.z * P.mom_kl;
    const int kend = kbeg + P.mom_kl < nz ? kbeg + P.mom_kl : nz;
    if (tid == 0) s_full = nz;
    __syncthreads();
    // the region columns this thread stages, and the levels full in all columns
    int gcol[NS];
#pragma unroll
    for (int q = 0; q < NS; ++q) {
        const int r = tid + q * NT;
        gcol[q] = -1;
        if (r < MOM_RN) {
            const int rj = r / MOM_RX, ri = r - rj * MOM_RX;
            gcol[q] = wrapi(j0 - 2 + rj, ny) * nx + wrapi(i0 - 2 + ri, nx);
            const int2 kfc = P.kface[gcol[q]];
            s_ku[r] = kfc.x;
            s_kv[r] = kfc.y;
            // a face at the region's edge has a column outside of it, which may be shallower
            int kf = P.kinfo[gcol[q]].x;
            if (kfc.x > 0) kf = min(kf, kfc.x + 1);
            if (kfc.y > 0) kf = min(kf, kfc.y + 1);
            if (kf < nz) atomicMin(&s_full, kf);
        }
    }
    // level k's u and v of the region go to buffer (k - kbeg) & 1; level k + 1's
    // copies are in flight while level k is computed
    auto stage = [&](int k) {
        const size_t o = (size_t)k * P.n2;
        const int buf = (k - kbeg) & 1;
#pragma unroll
        for (int q = 0; q < NS; ++q)
            if (gcol[q] >= 0) {
                cp_async_elem(&s_u[buf][tid + q * NT], u + o + gcol[q]);
                cp_async_elem(&s_v[buf][tid + q * NT], v + o + gcol[q]);
            }
        cp_async_commit();
    };
    stage(kbeg);
    // the next level's plane: every thread is done with the previous level, whose buffer
    // level k + 1 takes
    auto next_level = [&](int k) {
        __syncthreads();
        if (k + 1 < kend) {
            stage(k + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
    };
    const int rc = (ty + 2) * MOM_RX + tx + 2;
    const size_t n2 = (size_t)P.n2;
    const int wi = wrapi(i, nx), wj = wrapi(j, ny);
    const int c = wj * nx + wi;
    // the face's far column (east for u, north for v) and its wet levels
    const int cf = comp ? wrapi(j + 1, ny) * nx + wi : wj * nx + wrapi(i + 1, nx);
    const int kff = comp ? P.kface[c].y : P.kface[c].x;
    const real tau = comp ? P.tau_v[c] : P.tau_u[c];
    const real g2 = P.scheme != 2 ? real(comp ? gy2[c] : gx2[c]) : real(0.0);
    const real* __restrict__ X = comp ? v : u;
    auto Xc = [&](int kk) { return (kk >= 0 && kk < nz) ? X[(size_t)kk * n2 + c] : real(0.0); };
    MomCarry q{real(0.0), real(0.0), real(0.0), real(0.0), real(0.0)};
    if (live) {
        q.x_m1 = Xc(kbeg - 1);
        q.x_0 = Xc(kbeg);
        q.x_p1 = Xc(kbeg + 1);
        const size_t ob = (size_t)kbeg * n2;
        if (P.advection != 0)
            q.fz = mom_vflux(P, kbeg, kff, Xc(kbeg - 2), q.x_m1, q.x_0, q.x_p1, w[ob + c], w[ob + cf]);
        if (kbeg == 0) {
            q.df = tau;
        } else {
            const ColGeoR gc = ColGeoR::load(P, c), gf = ColGeoR::load(P, cf);
            real m, m3c, m3a;
            const real dz_m1 = face_dz(P, kff, kbeg - 1, gc.dz(P, kbeg - 1, m3a), gf.dz(P, kbeg - 1, m));
            const real dz_0 = face_dz(P, kff, kbeg, gc.dz(P, kbeg, m3c), gf.dz(P, kbeg, m));
            const real bot = (m3a > real(0.0) && m3c == real(0.0)) ? real(1.0) : real(0.0);
            q.df = diff_flux(km[ob + c], q.x_m1, q.x_0, dz_m1, dz_0, bot);
        }
    }
    __syncthreads();  // s_full
    // levels [kbeg, kfull) have full columns at themselves and the level below
    const int kfull = s_full - 1 < kend ? s_full - 1 : kend;
    int k = kbeg;
    if (k < kfull) {
        const unsigned fl = comp ? mom_face_flags(s_kv, s_ku, rc, MOM_RX, 1) : mom_face_flags(s_ku, s_kv, rc, 1, MOM_RX);
        for (; k < kfull; ++k) {
            next_level(k);
            if (!live) continue;
            const size_t o = (size_t)k * n2, at = o + c, af = o + cf;
            const int buf = (k - kbeg) & 1;
            const real x_p2 = k + 2 < nz ? X[at + 2 * n2] : real(0.0);
            const real K_1 = km[at + n2], w_c = w[at + n2], w_f = w[af + n2];
            const wide phc = phi[at], phf = phi[af], bc = b[at], bf = b[af];
            if (comp)
                mom_full_level<1>(P, s_v[buf] + rc, s_u[buf] + rc, fl, kff, k, x_p2, K_1, w_c, w_f, phc, phf, bc, bf,
                                  tau, g2, at, MomOut{pgy, avpu, dzv, stv, rv}, q);
            else
                mom_full_level<0>(P, s_u[buf] + rc, s_v[buf] + rc, fl, kff, k, x_p2, K_1, w_c, w_f, phc, phf, bc, bf,
                                  tau, g2, at, MomOut{pgx, avpv, dzu, stu, ru}, q);
        }
    }
    if (k >= kend) return;
    const ColGeoR gc = ColGeoR::load(P, c), gf = ColGeoR::load(P, cf);
#ifdef OC_MIXED
    // the pressure gradient's depths in fp64 (FP32 depths of ~4 km carry 2e-4 m errors)
    const ColGeo64 gc64 = ColGeo64::load(P, c), gf64 = ColGeo64::load(P, cf);
#endif
    // face thickness of the column's face at level kk (0 outside)
    auto dzf_at = [&](int kk) {
        if (kk < 0 || kk >= nz) return real(0.0);
        real m;
        return face_dz(P, kff, kk, gc.dz(P, kk, m), gf.dz(P, kk, m));
    };
    const MomOut out = comp ? MomOut{pgy, avpu, dzv, stv, rv} : MomOut{pgx, avpv, dzu, stu, ru};
    real dz_0 = dzf_at(k);
    for (; k < kend; ++k) {
        const size_t o = (size_t)k * n2;
        next_level(k);
        if (!live) continue;
        const int buf = (k - kbeg) & 1;
        const TileLevel lv{s_u[buf], s_v[buf], s_ku, s_kv, rc, k};
        const real x_p2 = Xc(k + 2);
        const real dz_p1 = dzf_at(k + 1);
        const real K_1 = km[o + n2 + c];
        real m3c, m3f;
        const real dz_c = gc.dz(P, k, m3c), dz_f = gf.dz(P, k, m3f);
        const real m3f_k = k < kff ? real(1.0) : real(0.0);
        const real bottom_k = (m3c > real(0.0) && k + 1 >= gc.kb) ? real(1.0) : real(0.0);
        // ---- pressure gradient at a common depth (model3d_v05.py:211-230), in
        // fp64 on both paths: it is a small difference of large potentials
        const wide phc = phi[o + c], phf = phi[o + cf];
        const wide bc = b[o + c], bf = b[o + cf];
        const wide dxy = comp ? P.dy64 : P.dx64;
        wide pgw;
        if (P.pgf_correction) {
#ifdef OC_MIXED
            const wide zc_c = gc64.above(P, k) + 0.5 * gc64.dz(P, k);
            const wide zc_f = gf64.above(P, k) + 0.5 * gf64.dz(P, k);
#else
            const wide zc_c = gc.above(P, k) + 0.5 * dz_c;
            const wide zc_f = gf.above(P, k) + 0.5 * dz_f;
#endif
            const wide zf = 0.5 * (zc_c + zc_f);
            pgw = m3f_k * ((phf + bf * (zf - zc_f)) - (phc + bc * (zf - zc_c))) / dxy;
        } else {
            pgw = m3f_k * (phf - phc) / dxy * m3f_k;
        }
        const real pg = real(pgw);
        out.pg[o + c] = pg;
        // ---- Coriolis average of the old state (v at u points, u at v points)
        const real av = comp ? u_on_v_at(lv) : v_on_u_at(lv);
        out.av[o + c] = av;
        // ---- explicit vertical diffusion: top flux carried, bottom flux formed here
        const real db = (k < nz - 1) ? diff_flux(K_1, q.x_0, q.x_p1, dz_0, dz_p1, bottom_k) : real(0.0);
        real dz;
        {
            const real mk = m3c > real(0.0) ? real(1.0) : real(0.0);
            const real id = inv_pos(dz_0);
            const real flux = (q.df - db) * id;
            const real drag = P.bottom_drag * q.x_0 * bottom_k;
            dz = (flux - drag * id) * mk;
        }
        out.dz[o + c] = dz;
        // ---- advection and horizontal viscosity, then the stress increment
        real ex = real(0.0), fb = real(0.0);
        if (P.advection != 0) {
            fb = mom_vflux(P, k + 1, kff, q.x_m1, q.x_0, q.x_p1, x_p2, w[o + n2 + c], w[o + n2 + cf]);
            const real a = (comp ? mom_adv_v_xy(P, lv) : mom_adv_u_xy(P, lv)) + (q.fz - fb) / P.dz_nom[k];
            ex = ex - a * m3f_k;
        }
        if (P.a_h > real(0.0)) {
            Nbr nb;
            nb.init(wi, wj, nx, ny);
            ex = ex + P.a_h * hlap(P, nb, X, k, comp);
        }
        const real st = (k == 0) ? P.thv_dt * tau * inv_pos(dz_0) + P.dt * ex : real(0.0) + P.dt * ex;
        out.st[o + c] = st;
        out.rhs[o + c] = predictor(P, q.x_0, comp ? P.neg_f0 : P.f0, av, av, pg, g2, m3f_k, dz, st);
        // roll down one level
        q.fz = fb;
        q.df = db;
        q.x_m1 = q.x_0;
        q.x_0 = q.x_p1;
        q.x_p1 = x_p2;
        dz_0 = dz_p1;
    }
}

// ------------------------------------------------------------------ predictor + column solves
// Per cell, for a Picard iteration after the first (whose right-hand sides
// k_mom_column forms): both right-hand sides with the iterate's Coriolis averages.
__global__ void __launch_bounds__(256) k_predictor_rhs(
    KPR P, const real* __restrict__ u, const real* __restrict__ v,
    const real* __restrict__ u_it, const real* __restrict__ v_it,
    const real* __restrict__ pgx, const real* __restrict__ pgy,
    const real* __restrict__ avpv, const real* __restrict__ avpu,
    const real* __restrict__ dzu, const real* __restrict__ dzv,
    const real* __restrict__ stu, const real* __restrict__ stv,
    const wide* __restrict__ gx2, const wide* __restrict__ gy2, real* __restrict__ ru,
    real* __restrict__ rv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y * blockDim.y + threadIdx.y;
    const int k = blockIdx.z;
    if (i >= P.nx || j >= P.ny) return;
    const int c = j * P.nx + i;
    const size_t o = (size_t)k * P.n2;
    Nbr nb;
    nb.init(i, j, P.nx, P.ny);
    const real it_v = v_on_u(P, nb, v_it, o, k), it_u = u_on_v(P, nb, u_it, o, k);
    const real g2x = P.scheme != 2 ? real(gx2[c]) : real(0.0), g2y = P.scheme != 2 ? real(gy2[c]) : real(0.0);
    ru[o + c] = predictor(P, u[o + c], P.f0, avpv[o + c], it_v, pgx[o + c], g2x, col_m3u(P, c, k), dzu[o + c],
                          stu[o + c]);
    rv[o + c] = predictor(P, v[o + c], P.neg_f0, avpu[o + c], it_u, pgy[o + c], g2y, col_m3v(P, c, k), dzv[o + c],
                          stv[o + c]);
}

// Per column: both momentum tridiagonals with the cell column's rows
// (vertical.py:17-44 on vertical_var.py:35-77 coefficients), the cell-mask
// multiply and the depth-integrated transports (model3d_v05.py:426-433). The
// right-hand sides arrive in gh_u/gh_v; the forward elimination overwrites them
// with its intermediate values, the back substitution with the solution, and
// the transports are summed in a last, downward pass to keep the reference's
// order. Only the elimination coefficients stay in the thread. The rows are divided out
// here: with the level table's reciprocals 512 x 512 x 50 takes 254 us a launch instead of
// 250 (FP32 175 and 167), 256 x 256 x 128 281 instead of 275 (FP32 218 and 206).
template <int NZM>
__global__ void __launch_bounds__(128) k_momentum_solve(KPR P, const real* __restrict__ km,
                                                        real* __restrict__ ghu,
                                                        real* __restrict__ ghv,
                                                        wide* __restrict__ Ug,
                                                        wide* __restrict__ Vg) {
    COLUMN_PROLOGUE
    const int nz = P.nz;
    const int c = nb.c;
    const ColGeoR g = ColGeoR::load(P, c);
    real cs[NZM];
    real m3_k, dz_k = g.dz(P, 0, m3_k);
    real dzi_k = dz_k;
    real km_k = km[c];
    real du = real(0.0), dv = real(0.0), cp = real(0.0);
#pragma unroll 4
    for (int k = 0; k < nz; ++k) {
        const size_t o = (size_t)k * n2 + c;
        const real km_k1 = km[o + n2];
        const real ru = ghu[o], rv = ghv[o];
        real m3_k1 = real(0.0), dz_k1 = real(0.0);
        if (k + 1 < nz) dz_k1 = g.dz(P, k + 1, m3_k1);
        const real dzi_k1 = (k + 1 < nz) ? real(0.5) * (dz_k + dz_k1) : dz_k;
        real sub, diag, sup;
        implicit_row(P, k, dz_k, m3_k, m3_k1, dzi_k, dzi_k1, km_k, km_k1, P.thv_dt_drag, sub, diag, sup);
        if (k == 0) {
            cp = sup / diag;
            du = ru / diag;
            dv = rv / diag;
        } else {
            const real den = diag - sub * cp;
            cp = sup / den;
            du = (ru - sub * du) / den;
            dv = (rv - sub * dv) / den;
        }
        cs[k] = cp;
        ghu[o] = du;
        ghv[o] = dv;
        km_k = km_k1;
        dz_k = dz_k1;
        m3_k = m3_k1;
        dzi_k = dzi_k1;
    }
    real xu = du, xv = dv;
    {
        const size_t o = (size_t)(nz - 1) * n2 + c;
        const real m = (nz - 1 < g.kb) ? real(1.0) : real(0.0);
        ghu[o] = xu * m;
        ghv[o] = xv * m;
    }
#pragma unroll 4
    for (int k = nz - 2; k >= 0; --k) {
        const size_t o = (size_t)k * n2 + c;
        const real m = (k < g.kb) ? real(1.0) : real(0.0);
        xu = ghu[o] - cs[k] * xu;
        xv = ghv[o] - cs[k] * xv;
        ghu[o] = xu * m;
        ghv[o] = xv * m;
    }
    const ColGeoR ge = ColGeoR::load(P, nb.at(0, 1)), gn = ColGeoR::load(P, nb.at(1, 0));
    const int2 kfc = P.kface[c];
    wide su = 0.0, sv = 0.0;  // depth sums in fp64 on both paths
#pragma unroll 4
    for (int k = 0; k < nz; ++k) {
        const size_t o = (size_t)k * n2 + c;
        real m3c, m3e, m3n;
        const real dzc = g.dz(P, k, m3c);
        const real dze = ge.dz(P, k, m3e);
        const real dzn = gn.dz(P, k, m3n);
        const real tu = (k < kfc.x ? real(1.0) : real(0.0)) * face_combine(P, dzc, dze) * ghu[o];
        const real tv = (k < kfc.y ? real(1.0) : real(0.0)) * face_combine(P, dzc, dzn) * ghv[o];
        su = (k == 0) ? wide(tu) : su + wide(tu);
        sv = (k == 0) ? wide(tv) : sv + wide(tv);
    }
    Ug[c] = su;
    Vg[c] = sv;
}

// The same for one component per thread (threadIdx.z), for few columns: a level's chain has
// two divisions instead of three, and there are twice the warps. Each thread keeps the
// elimination coefficients, so on a large grid it is the slower form. us a launch by
// columns and by components: 16,384 x 50 60 and 51, 512 x 32 33 and 23, 46,937 x 37 39 and 31,
// 65,536 x 32 52 and 48, 122,880 x 30 67 and 84.
template <int NZM>
__global__ void __launch_bounds__(128) k_momentum_solve_few(KLR P, const real* __restrict__ km,
                                                            real* __restrict__ ghu, real* __restrict__ ghv,
                                                            wide* __restrict__ Ug, wide* __restrict__ Vg) {
    COLUMN_PROLOGUE
    const int nz = P.nz;
    const int c = nb.c;
    const bool comp = threadIdx.z;
    const ColGeoR g = ColGeoR::load(P, c);
    real* __restrict__ gh = comp ? ghv : ghu;
    real cs[NZM];
    real rdzi_k = g.rdz(P, 0);
    real km_k = km[c];
    real x = real(0.0), cp = real(0.0);
#pragma unroll 4
    for (int k = 0; k < nz; ++k) {
        const size_t o = (size_t)k * n2 + c;
        const real km_k1 = km[o + n2];
        const real r = gh[o];
        const real m3_k = k < g.kb ? real(1.0) : real(0.0), m3_k1 = k + 1 < g.kb ? real(1.0) : real(0.0);
        const real rdzi_k1 = (k + 1 < nz) ? g.rdzi(P, k + 1) : real(0.0);
        real sub, diag, sup;
        implicit_row_inv(P, k, g.rdz(P, k), m3_k, m3_k1, rdzi_k, rdzi_k1, km_k, km_k1, P.thv_dt_drag, sub, diag, sup);
        if (k == 0) {
            cp = sup / diag;
            x = r / diag;
        } else {
            const real den = diag - sub * cp;
            cp = sup / den;
            x = (r - sub * x) / den;
        }
        cs[k] = cp;
        gh[o] = x;
        km_k = km_k1;
        rdzi_k = rdzi_k1;
    }
    gh[(size_t)(nz - 1) * n2 + c] = x * ((nz - 1 < g.kb) ? real(1.0) : real(0.0));
#pragma unroll 4
    for (int k = nz - 2; k >= 0; --k) {
        const size_t o = (size_t)k * n2 + c;
        x = gh[o] - cs[k] * x;
        gh[o] = x * ((k < g.kb) ? real(1.0) : real(0.0));
    }
    const ColGeoR gf = ColGeoR::load(P, comp ? nb.at(1, 0) : nb.at(0, 1));
    const int kf = comp ? P.kface[c].y : P.kface[c].x;
    wide sum = 0.0;  // depth sum in fp64 on both paths
#pragma unroll 4
    for (int k = 0; k < nz; ++k) {
        real m3c, m3f;
        const real dzc = g.dz(P, k, m3c);
        const real dzf = gf.dz(P, k, m3f);
        const real t = (k < kf ? real(1.0) : real(0.0)) * face_combine(P, dzc, dzf) * gh[(size_t)k * n2 + c];
        sum = (k == 0) ? wide(t) : sum + wide(t);
    }
    (comp ? Vg : Ug)[c] = sum;
}

// ------------------------------------------------------------------ back substitution
// u = (gh_u - g dt theta q dx(eta_new) m3u) m3   (model3d_v05.py:404-406)
__global__ void k_backsub(KPR P, const real* __restrict__ ghu, const real* __restrict__ ghv,
                          const real* __restrict__ q, const wide* __restrict__ eta_new,
                          real* __restrict__ u_out, real* __restrict__ v_out) {
    COLUMN_PROLOGUE
    const size_t c = nb.c, ce = nb.at(0, 1), cn = nb.at(1, 0);
    // the surface gradient in fp64 on both paths (a difference of neighbouring elevations)
    const real gx = real(P.mask_u64[c] * (eta_new[ce] - eta_new[c]) / P.dx64);
    const real gy = real(P.mask_v64[c] * (eta_new[cn] - eta_new[c]) / P.dy64);
    const int kb = P.kinfo[c].y;
    const int2 kf = P.kface[c];
#pragma unroll 4
    for (int k = 0; k < P.nz; ++k) {
        const size_t o = (size_t)k * n2 + c;
        const real m3 = k < kb ? real(1.0) : real(0.0);
        const real m3u_k = k < kf.x ? real(1.0) : real(0.0);
        const real m3v_k = k < kf.y ? real(1.0) : real(0.0);
        const real qk = q[o];
        u_out[o] = (ghu[o] - P.c2 * qk * gx * m3u_k) * m3;
        v_out[o] = (ghv[o] - P.c2 * qk * gy * m3v_k) * m3;
    }
}

// the same by levels, for few columns
__global__ void __launch_bounds__(LV_X * LV_Y) k_backsub_few(KPR P, const real* __restrict__ ghu,
                                                         const real* __restrict__ ghv, const real* __restrict__ q,
                                                         const wide* __restrict__ eta_new, real* __restrict__ u_out,
                                                         real* __restrict__ v_out) {
    LEVELS_PROLOGUE
    if (!live) return;
    const size_t c = nb.c, ce = nb.at(0, 1), cn = nb.at(1, 0);
    // the surface gradient in fp64 on both paths (a difference of neighbouring elevations)
    const real gx = real(P.mask_u64[c] * (eta_new[ce] - eta_new[c]) / P.dx64);
    const real gy = real(P.mask_v64[c] * (eta_new[cn] - eta_new[c]) / P.dy64);
    const int kb = P.kinfo[c].y;
    const int2 kf = P.kface[c];
#pragma unroll 4
    for (int k = threadIdx.y; k < P.nz; k += LV_Y) {
        const size_t o = (size_t)k * n2 + c;
        const real m3 = k < kb ? real(1.0) : real(0.0);
        const real m3u_k = k < kf.x ? real(1.0) : real(0.0);
        const real m3v_k = k < kf.y ? real(1.0) : real(0.0);
        const real qk = q[o];
        u_out[o] = (ghu[o] - P.c2 * qk * gx * m3u_k) * m3;
        v_out[o] = (ghv[o] - P.c2 * qk * gy * m3v_k) * m3;
    }
}

// ------------------------------------------------------------------ tracers + EOS
// Tiled right-hand sides of the implicit tracer solves (model3d_v05.py:466-512).
// A CTA owns a TRX x TRY tile of columns and P.tr_kl levels and marches down the
// levels. At each level the horizontal face fluxes of the tile -- TRX + 1 east
// faces per row, TRY + 1 north faces per column -- are formed once into shared
// memory, the level below it staged meanwhile; a per-cell form would form
// every face twice, once from each side. The vertical face at the bottom of a
// cell is carried to the next level as the face at its top, and the column's
// tracer values, w and K_h roll in registers. Every face and cell value is
// formed by the reference's operations in the reference's order.
// Bound by instruction issue: the levels that are wet and full in every column of the tile
// and its ring, most of them over a flat bottom, take thicknesses and reciprocals from the
// level table and need no mask but the open faces. 512 x 512 x 50: 887 us a launch with one
// form for all levels, 694 with the short one above the general one (FP32 548, now 438).
constexpr int TRX = 32, TRY = 8;

// tracer value on interface kk of a column (0 = surface) from the column values
// at kk-2, kk-1, kk, kk+1 and w there (model3d_v05.py:502-510)
__device__ __forceinline__ real tracer_vface(const KPR& P, const ColGeoR& g, int kk, real f_m2, real f_m1,
                                               real f_0, real f_p1, real wv) {
    const int nz = P.nz;
    if (kk == 0) return f_0;
    if (kk == nz) return real(0.0);
    if (P.advection >= 3) {
        const real fu = (kk >= 2) ? f_m2 : real(0.0);
        const real fd = (kk + 1 <= nz - 1) ? f_p1 : real(0.0);
        const bool hu = (kk >= 2) && kk - 2 < g.kb;
        const bool hd = (kk + 1 <= nz - 1) && kk + 1 < g.kb;
        return kappa_face_z(P, fu, f_m1, f_0, fd, wv, hu, hd, P.advection == 4);
    }
    return real(0.5) * (f_m1 + f_0);
}

__global__ void __launch_bounds__(TRX * TRY, OC_MINB_TRACER) k_tracer_rhs(KLR P, const real* __restrict__ C0,
                                                             const real* __restrict__ S,
                                                             const real* __restrict__ u,
                                                             const real* __restrict__ v,
                                                             const real* __restrict__ w,
                                                             const real* __restrict__ kh,
                                                             real* __restrict__ rT,
                                                             real* __restrict__ rS) {
    // C0 is T with TS tracers, else the buoyancy (the fp64 path's only tracer).
    // The tile's columns plus a 2-column ring: flat 2D index and compact geometry
    // (once), then each level's tracers and face velocities (staged per level)
    constexpr int RX = TRX + 4, RY = TRY + 4, RNC = RX * RY;
    // level indices are at most 128: the column's (kf, kb) and its faces' wet
    // levels (ku, kv) fit one byte each
    __shared__ int s_g[RNC];
    __shared__ uchar4 s_k[RNC];
    __shared__ real s_d0[RNC], s_d1[RNC];
    // level planes, double-buffered: [buffer][field] tracers, [buffer] face velocities
    __shared__ real s_f[2][2][RNC], s_u[2][RNC], s_v[2][RNC];
    __shared__ int s_full;  // levels that are full in every column of the region
    __shared__ real sfx[2][TRY][TRX + 1];  // [field][row][west face of column]
    __shared__ real sfy[2][TRY + 1][TRX];  // [field][south face of row][column]
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int tid = ty * TRX + tx;
    const int i0 = blockIdx.x * TRX, j0 = blockIdx.y * TRY;
    const int i = i0 + tx, j = j0 + ty;
    const int nx = P.nx, ny = P.ny, nz = P.nz;
    const size_t n2 = P.n2;
    const bool live = i < nx && j < ny;
    const bool ts = P.tracers_ts;
    const int nf = ts ? 2 : 1;
    const bool adv = P.advection != 0;
    const int kbeg = blockIdx.z * P.tr_kl;
    const int kend = kbeg + P.tr_kl < nz ? kbeg + P.tr_kl : nz;
    // faces this thread forms: the west and south faces of its cell, and for two
    // warps the east faces of the tile's last column / north faces of its last row
    const bool xextra = ty == TRY - 2 && tx < TRY, yextra = ty == TRY - 1;
    const int c = wrapi(j, ny) * nx + wrapi(i, nx);
    const ColGeoR g = ColGeoR::load(P, c);
    real* __restrict__ R0 = rT;
    if (tid == 0) s_full = nz;
    __syncthreads();
    for (int r = tid; r < RNC; r += TRX * TRY) {
        const int rj = r / RX, ri = r - rj * RX;
        const int gc = wrapi(j0 - 2 + rj, ny) * nx + wrapi(i0 - 2 + ri, nx);
        const int2 ki = P.kinfo[gc], kfc = P.kface[gc];
        const auto dx = P.dzx[gc];
        s_g[r] = gc;
        s_k[r] = make_uchar4((unsigned char)ki.x, (unsigned char)ki.y, (unsigned char)kfc.x, (unsigned char)kfc.y);
        s_d0[r] = dx.x;
        s_d1[r] = dx.y;
        if (ki.x < nz) atomicMin(&s_full, ki.x);
    }
    // thickness and wet flag of region column r at level k (col_dz from the staged geometry)
    auto sdz = [&](int r, int k, real& m3) {
        const uchar4 q = s_k[r];
        if (k >= q.y) {
            m3 = real(0.0);
            return real(0.0);
        }
        m3 = real(1.0);
        if (k < q.x) return P.dzr[k];
        return k == q.x ? s_d0[r] : s_d1[r];
    };
    // flux through a face with stencil cells (cm, c0, c1, cp) of the region,
    // normal velocity vel and face wet levels kfa: face thickness x velocity x face value
    // (model3d_v05.py:482-501)
    auto sflux = [&](const real* F, int cm, int c0, int c1, int cp, real vel, int kfa, int k) {
        real m;
        const real dzf = face_dz(P, kfa, k, sdz(c0, k, m), sdz(c1, k, m));
        const real a = F[c0], b = F[c1];
        real val;
        if (P.advection == 1)
            val = real(0.5) * (a + b);
        else if (P.advection >= 3)
            val = kappa_face(P, F[cm], a, b, F[cp], vel, k < s_k[cm].y ? real(1.0) : real(0.0),
                             k < s_k[cp].y ? real(1.0) : real(0.0), P.advection == 4);
        else
            val = vel > real(0.0) ? a : b;
        return dzf * vel * val;
    };
    const int rc = (ty + 2) * RX + tx + 2;                    // this thread's cell in the region
    const int rce = (tx + 2) * RX + TRX + 1;                  // east-column cell of row tx (x extras)
    const int rcn = (TRY + 1) * RX + tx + 2;                  // north-row cell of column tx (y extras)
    // rolling column values of each field at k-1, k, k+1 and the face at the top of level k
    real fm1[2] = {real(0.0), real(0.0)}, f0[2] = {real(0.0), real(0.0)}, fp1[2] = {real(0.0), real(0.0)}, ftop[2] = {real(0.0), real(0.0)};
    real w_k = real(0.0), kh_k = real(0.0);
    if (live) {
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            if (f >= nf) break;
            const real* __restrict__ C = f == 0 ? C0 : S;
            const real fm2 = kbeg >= 2 ? C[(size_t)(kbeg - 2) * n2 + c] : real(0.0);
            fm1[f] = kbeg >= 1 ? C[(size_t)(kbeg - 1) * n2 + c] : real(0.0);
            f0[f] = C[(size_t)kbeg * n2 + c];
            fp1[f] = kbeg + 1 < nz ? C[(size_t)(kbeg + 1) * n2 + c] : real(0.0);
            if (adv) ftop[f] = tracer_vface(P, g, kbeg, fm2, fm1[f], f0[f], fp1[f], w[(size_t)kbeg * n2 + c]);
        }
        w_k = w[(size_t)kbeg * n2 + c];
        kh_k = kh[(size_t)kbeg * n2 + c];
    }
    // level k's planes go to buffer (k - kbeg) & 1; level k + 1's copies are in
    // flight while level k is computed (each thread copies the region cells
    // whose s_g it wrote itself)
    auto stage = [&](int k) {
        const size_t o = (size_t)k * n2;
        const int buf = (k - kbeg) & 1;
        for (int r = tid; r < RNC; r += TRX * TRY) {
            const size_t g = o + s_g[r];
            cp_async_elem(&s_f[buf][0][r], C0 + g);
            if (ts) cp_async_elem(&s_f[buf][1][r], S + g);
            cp_async_elem(&s_u[buf][r], u + g);
            cp_async_elem(&s_v[buf][r], v + g);
        }
        cp_async_commit();
    };
    // the level's plane in place, level k + 1's on its way: every thread is done with the
    // previous level, whose buffer level k + 1 takes
    auto next_level = [&](int k) {
        __syncthreads();
        if (k + 1 < kend) {
            stage(k + 1);
            cp_async_wait<1>();
        } else {
            cp_async_wait<0>();
        }
        __syncthreads();
    };
    if (adv) stage(kbeg);
    __syncthreads();  // s_full
    // Levels [kbeg, kfull): every column of the region is wet and full there and one level
    // below. Thicknesses and their reciprocals come from the level table, every far cell
    // is wet, a face has the level's thickness or none (fl: open west, south, east and
    // north faces of the cell; of the extra faces, the one this thread forms), and the
    // diffusive flux at a cell's bottom is carried to the next level's top as the
    // advective face is. The values are the general form's, operation for operation.
    int k = kbeg;
    const int kfull = s_full - 1 < kend ? s_full - 1 : kend;
    if (k < kfull) {
        const unsigned fl = (s_k[rc - 1].z > 0 ? 1u : 0u) | (s_k[rc - RX].w > 0 ? 2u : 0u) |
                            (s_k[rc].z > 0 ? 4u : 0u) | (s_k[rc].w > 0 ? 8u : 0u);
        const bool xopen = xextra && s_k[rce].z > 0, yopen = yextra && s_k[rcn].w > 0;
        real dtop[2] = {real(0.0), real(0.0)};  // diffusive flux through the top of level k
        if (live)
#pragma unroll
            for (int f = 0; f < 2; ++f)
                dtop[f] = k == 0 ? (ts ? (f == 0 ? P.flux_t : P.flux_s) : real(0.0))
                                 : kh_k * (fm1[f] - f0[f]) * P.rdzi[k];
        // flux through a face whose upstream-side and downstream-side cells are c0 and c0 + st
        auto fflux = [&](const real* F, int c0, int st, real vel, real dzf) {
            const real a = F[c0], b = F[c0 + st];
            real val;
            if (P.advection == 1) val = real(0.5) * (a + b);
            else if (P.advection >= 3) val = kappa_face_f(P, F[c0 - st], a, b, F[c0 + 2 * st], vel, true, true, P.advection == 4);
            else val = vel > real(0.0) ? a : b;
            return dzf * vel * val;
        };
        for (; k < kfull; ++k) {
            const size_t o = (size_t)k * n2;
            const int buf = (k - kbeg) & 1;
            if (adv) {
                next_level(k);
                const real* su = s_u[buf];
                const real* sv = s_v[buf];
                const real dzf = P.fdz[k];
#pragma unroll 1
                for (int f = 0; f < nf; ++f) {
                    const real* F = s_f[buf][f];
                    sfx[f][ty][tx] = fflux(F, rc - 1, 1, su[rc - 1], fl & 1 ? dzf : real(0.0));
                    sfy[f][ty][tx] = fflux(F, rc - RX, RX, sv[rc - RX], fl & 2 ? dzf : real(0.0));
                    if (xextra) sfx[f][tx][TRX] = fflux(F, rce, 1, su[rce], xopen ? dzf : real(0.0));
                    if (yextra) sfy[f][TRY][tx] = fflux(F, rcn, RX, sv[rcn], yopen ? dzf : real(0.0));
                }
                __syncthreads();
            }
            if (!live) continue;
            const real w_k1 = w[o + n2 + c];
            const real kh_k1 = kh[o + n2 + c];
            const real inv = P.rdz[k];
#pragma unroll
            for (int f = 0; f < 2; ++f) {
                if (f >= nf) break;
                const real* __restrict__ C = f == 0 ? C0 : S;
                const real fp2 = (k + 2 < nz) ? C[o + 2 * n2 + c] : real(0.0);
                const real surf = ts ? (f == 0 ? P.flux_t : P.flux_s) : real(0.0);
                real tend = ts ? real(0.0) : P.neg_n2 * (real(0.5) * (w_k + w_k1));
                real fbot = real(0.0);
                if (adv) {
                    fbot = tracer_vface(P, g, k + 1, fm1[f], f0[f], fp1[f], fp2, w_k1);
                    const real hdiv = ((sfx[f][ty][tx + 1] - sfx[f][ty][tx]) / P.dx +
                                       (sfy[f][ty + 1][tx] - sfy[f][ty][tx]) / P.dy) * inv;
                    const real vdiv = (w_k * ftop[f] - w_k1 * fbot) * inv;
                    tend = tend - (hdiv + vdiv);
                }
                if (P.k_h > real(0.0)) {
                    // hlap with the level's open faces; F from global memory, as the tile is staged
                    // only with advection
                    const int ce = wrapi(j, ny) * nx + wrapi(i + 1, nx), cw = wrapi(j, ny) * nx + wrapi(i - 1, nx);
                    const int cn = wrapi(j + 1, ny) * nx + wrapi(i, nx), cs = wrapi(j - 1, ny) * nx + wrapi(i, nx);
                    const real gx0 = (fl & 4 ? real(1.0) : real(0.0)) * (C[o + ce] - f0[f]) / P.dx;
                    const real gxw = (fl & 1 ? real(1.0) : real(0.0)) * (f0[f] - C[o + cw]) / P.dx;
                    const real gy0 = (fl & 8 ? real(1.0) : real(0.0)) * (C[o + cn] - f0[f]) / P.dy;
                    const real gys = (fl & 2 ? real(1.0) : real(0.0)) * (f0[f] - C[o + cs]) / P.dy;
                    tend = tend + P.k_h * ((gx0 - gxw) / P.dx + (gy0 - gys) / P.dy);
                }
                const real dbot = kh_k1 * (f0[f] - fp1[f]) * P.rdzi[k + 1];
                const real diff = (dtop[f] - dbot) * inv;
                real rhs = f0[f] + P.dt * tend + P.c3 * diff;
                if (k == 0) rhs = rhs + P.thv_dt * surf * inv;
                (f == 0 ? R0 : rS)[o + c] = rhs;
                dtop[f] = dbot;
                ftop[f] = fbot;
                fm1[f] = f0[f];
                f0[f] = fp1[f];
                fp1[f] = fp2;
            }
            w_k = w_k1;
            kh_k = kh_k1;
        }
    }
    for (; k < kend; ++k) {
        const size_t o = (size_t)k * n2;
        if (adv) {
            next_level(k);
            const int buf = (k - kbeg) & 1;
            const real* su = s_u[buf];
            const real* sv = s_v[buf];
#pragma unroll 1
            for (int f = 0; f < nf; ++f) {
                const real* F = s_f[buf][f];
                // west face of this cell (cells rc-2 .. rc+1), south face (rc-2RX .. rc+RX)
                sfx[f][ty][tx] = sflux(F, rc - 2, rc - 1, rc, rc + 1, su[rc - 1], s_k[rc - 1].z, k);
                sfy[f][ty][tx] = sflux(F, rc - 2 * RX, rc - RX, rc, rc + RX, sv[rc - RX], s_k[rc - RX].w, k);
                if (xextra) sfx[f][tx][TRX] = sflux(F, rce - 1, rce, rce + 1, rce + 2, su[rce], s_k[rce].z, k);
                if (yextra)
                    sfy[f][TRY][tx] = sflux(F, rcn - RX, rcn, rcn + RX, rcn + 2 * RX, sv[rcn], s_k[rcn].w, k);
            }
            __syncthreads();
        }
        if (!live) continue;
        real m3k, m3_m1 = real(0.0), m3_p1 = real(0.0);
        const real dzk = g.dz(P, k, m3k);
        const real dz_m1 = (k > 0) ? g.dz(P, k - 1, m3_m1) : real(0.0);
        const real dz_p1 = (k + 1 < nz) ? g.dz(P, k + 1, m3_p1) : real(0.0);
        const real bottom_m1 = (k > 0 && m3_m1 > real(0.0) && m3k == real(0.0)) ? real(1.0) : real(0.0);
        const real bottom_k = (m3k > real(0.0) && m3_p1 == real(0.0)) ? real(1.0) : real(0.0);
        const real w_k1 = w[o + n2 + c];
        const real kh_k1 = kh[o + n2 + c];
        const real inv = inv_pos(dzk);
#pragma unroll
        for (int f = 0; f < 2; ++f) {
            if (f >= nf) break;
            const real* __restrict__ C = f == 0 ? C0 : S;
            const real fp2 = (k + 2 < nz) ? C[o + 2 * n2 + c] : real(0.0);
            const real surf = ts ? (f == 0 ? P.flux_t : P.flux_s) : real(0.0);
            real tend = ts ? real(0.0) : P.neg_n2 * (real(0.5) * (w_k + w_k1));
            real fbot = real(0.0);
            if (adv) {
                fbot = tracer_vface(P, g, k + 1, fm1[f], f0[f], fp1[f], fp2, w_k1);
                const real hdiv = ((sfx[f][ty][tx + 1] - sfx[f][ty][tx]) / P.dx +
                                     (sfy[f][ty + 1][tx] - sfy[f][ty][tx]) / P.dy) *
                                    inv;
                const real vdiv = (w_k * ftop[f] - w_k1 * fbot) * inv;
                tend = tend - (hdiv + vdiv) * m3k;
            }
            if (P.k_h > real(0.0)) {
                Nbr nb;
                nb.init(wrapi(i, nx), wrapi(j, ny), nx, ny);
                tend = tend + P.k_h * hlap(P, nb, C, k, 2);
            }
            // explicit vertical diffusion with zero drag (vertical_var.py:80-106)
            const real diff = explicit_dz(P, k, k > 0 ? fm1[f] : real(0.0), f0[f], k + 1 < nz ? fp1[f] : real(0.0), kh_k,
                                            kh_k1, dz_m1, dzk, dz_p1, bottom_m1, bottom_k, m3k, surf, real(0.0));
            real rhs = f0[f] + P.dt * tend + P.c3 * diff;
            if (k == 0) rhs = rhs + P.thv_dt * surf * inv_pos(dzk);
            (f == 0 ? R0 : rS)[o + c] = rhs;
            ftop[f] = fbot;
            fm1[f] = f0[f];
            f0[f] = fp1[f];
            fp1[f] = fp2;
        }
        w_k = w_k1;
        kh_k = kh_k1;
    }
}

// One thread per column: the implicit solves with the diffusivity rows
// (shared by T and S), the cell mask, and the EOS of the new T/S
// (model3d_v05.py:514-533). The forward elimination stores its right-hand sides
// in the outputs; the back substitution finishes each level there, EOS
// included, with the level-centre depth in closed form (col_above is the
// sequential sum of the thicknesses above, bit for bit). The rows are divided out here, as in
// k_momentum_solve: with the level table's reciprocals 256 x 256 x 128 takes 312 us instead of
// 305 (FP32 267 and 256), 512 x 512 x 50 311 and 312 (FP32 239 and 233).
template <int NZM>
__global__ void __launch_bounds__(128) k_tracer_solve(KPR P, const real* __restrict__ rT,
                                                      const real* __restrict__ rS,
                                                      const real* __restrict__ kh,
                                                      real* __restrict__ T_out,
                                                      real* __restrict__ S_out,
                                                      wide* __restrict__ b_out) {
    COLUMN_PROLOGUE
    const int nz = P.nz;
    const int c = nb.c;
    const ColGeoR g = ColGeoR::load(P, c);
    real cs[NZM];
    const bool ts = P.tracers_ts;
#ifdef OC_MIXED
    real* __restrict__ o1 = T_out;  // the mixed path carries T and S (checked on the host)
    const ColGeo64 g64 = ColGeo64::load(P, c);
#else
    real* __restrict__ o1 = ts ? T_out : b_out;
#endif
    real m3_k, dz_k = g.dz(P, 0, m3_k);
    real dzi_k = dz_k;
    real kh_k = kh[c];
    real d1 = real(0.0), d2 = real(0.0), cp = real(0.0);
#pragma unroll 4
    for (int k = 0; k < nz; ++k) {
        const size_t o = (size_t)k * n2 + c;
        const real kh_k1 = kh[o + n2];
        real m3_k1 = real(0.0), dz_k1 = real(0.0);
        if (k + 1 < nz) dz_k1 = g.dz(P, k + 1, m3_k1);
        const real dzi_k1 = (k + 1 < nz) ? real(0.5) * (dz_k + dz_k1) : dz_k;
        const real r1 = rT[o];
        const real r2 = ts ? rS[o] : real(0.0);
        real sub, diag, sup;
        implicit_row(P, k, dz_k, m3_k, m3_k1, dzi_k, dzi_k1, kh_k, kh_k1, P.thv_dt_zero, sub, diag, sup);
        if (k == 0) {
            cp = sup / diag;
            d1 = r1 / diag;
            d2 = r2 / diag;
        } else {
            const real den = diag - sub * cp;
            cp = sup / den;
            d1 = (r1 - sub * d1) / den;
            d2 = (r2 - sub * d2) / den;
        }
        cs[k] = cp;
        if (k + 1 < nz) {
            o1[o] = d1;
            if (ts) S_out[o] = d2;
        }
        kh_k = kh_k1;
        dz_k = dz_k1;
        m3_k = m3_k1;
        dzi_k = dzi_k1;
    }
    real x1 = d1, x2 = d2;
#pragma unroll 4
    for (int k = nz - 1; k >= 0; --k) {
        const size_t o = (size_t)k * n2 + c;
        if (k < nz - 1) {
            x1 = o1[o] - cs[k] * x1;
            if (ts) x2 = S_out[o] - cs[k] * x2;
        }
        real m3;
        const real dz = g.dz(P, k, m3);
        if (ts) {
            const real Tn = x1 * m3;
            const real Sn = x2 * m3;
#ifdef OC_MIXED
            const wide zc = g64.above(P, k) + 0.5 * g64.dz(P, k);
#else
            const wide zc = col_above(P, c, k) + real(0.5) * dz;
#endif
            T_out[o] = Tn;
            S_out[o] = Sn;
            b_out[o] = buoyancy_of(P, wide(Tn), wide(Sn), zc) * wide(m3);  // EOS in fp64 on both paths
        } else {
            b_out[o] = wide(x1 * m3);
        }
    }
}

// The same by levels, for few columns: a CTA takes SL_X columns of a row with SL_Y threads
// each, which form the column's rows side by side in shared memory and, after the
// elimination by a lane per column and field, its levels' EOS. us a launch by columns and
// by levels: 16,384 x 50 65 and 44, 512 x 32 13.6 and 5.6, 46,937 x 37 38 and 35, 65,536 x 32 75
// and 77, 262,144 x 50 306 and 448. (The momentum solve in this form gains at 16,384 and loses
// from 32,000 on.)
constexpr int SL_X = 32, SL_Y = 8;

struct SolveRows {  // of the thread's column, level k at [k * SL_X]
    real *sub, *dia, *sup, *r[2];
    __device__ __forceinline__ SolveRows(unsigned char* s, int nz, int col) {
        sub = reinterpret_cast<real*>(s) + col;
        dia = sub + nz * SL_X;
        sup = dia + nz * SL_X;
        r[0] = sup + nz * SL_X;
        r[1] = r[0] + nz * SL_X;
    }
};

// Forward elimination and back substitution of all the CTA's columns, by its first two
// warps: 16 columns each, the lanes of a warp's halves for the two right-hand sides. The
// halves form the same coefficients and store them in the place of sup.
__device__ __forceinline__ void solve_pairs(unsigned char* s, int nz) {
    if (threadIdx.y >= 2) return;
    const int lane = threadIdx.x;
    const SolveRows R(s, nz, threadIdx.y * 16 + (lane & 15));
    real* r = lane < 16 ? R.r[0] : R.r[1];
    real cp = real(0.0), x = real(0.0);
#pragma unroll 2
    for (int k = 0; k < nz; ++k) {
        const real sub = R.sub[k * SL_X], dia = R.dia[k * SL_X], sup = R.sup[k * SL_X], y = r[k * SL_X];
        __syncwarp();  // both halves have read sup
        if (k == 0) {
            cp = sup / dia;
            x = y / dia;
        } else {
            const real den = dia - sub * cp;
            cp = sup / den;
            x = (y - sub * x) / den;
        }
        R.sup[k * SL_X] = cp;
        r[k * SL_X] = x;
    }
    __syncwarp();
#pragma unroll 4
    for (int k = nz - 2; k >= 0; --k) {
        x = r[k * SL_X] - R.sup[k * SL_X] * x;
        r[k * SL_X] = x;
    }
}

// the rows of level k of a column (implicit_row_inv)
__device__ __forceinline__ void solve_row(const KLR& P, const ColGeoR& g, int k, real k_top, real k_bot, real drag,
                                          const SolveRows& R) {
    const real m3_k = k < g.kb ? real(1.0) : real(0.0), m3_k1 = k + 1 < g.kb ? real(1.0) : real(0.0);
    const real rdzi_k = k == 0 ? g.rdz(P, 0) : g.rdzi(P, k), rdzi_k1 = k + 1 < P.nz ? g.rdzi(P, k + 1) : real(0.0);
    real sub, diag, sup;
    implicit_row_inv(P, k, g.rdz(P, k), m3_k, m3_k1, rdzi_k, rdzi_k1, k_top, k_bot, drag, sub, diag, sup);
    R.sub[k * SL_X] = sub;
    R.dia[k * SL_X] = diag;
    R.sup[k * SL_X] = sup;
}

__global__ void __launch_bounds__(SL_X * SL_Y, 3) k_tracer_levels(KLR P, const real* __restrict__ rT,
                                                                 const real* __restrict__ rS,
                                                                 const real* __restrict__ kh, real* __restrict__ T_out,
                                                                 real* __restrict__ S_out, wide* __restrict__ b_out) {
    extern __shared__ __align__(16) unsigned char s_dyn[];
    const int tiles = (P.nx + SL_X - 1) / SL_X;
    const int j = blockIdx.x / tiles, i_own = (blockIdx.x - j * tiles) * SL_X + threadIdx.x;
    const bool live = i_own < P.nx;  // the others repeat the last column and store nothing
    const int i = live ? i_own : P.nx - 1, nz = P.nz, first = threadIdx.y;
    const size_t n2 = (size_t)P.n2;
    const int c = j * P.nx + i;
    const ColGeoR g = ColGeoR::load(P, c);
    const SolveRows R(s_dyn, nz, threadIdx.x);
    const bool ts = P.tracers_ts;
#pragma unroll 2
    for (int k = first; k < nz; k += SL_Y) {
        const size_t o = (size_t)k * n2 + c;
        const real r1 = rT[o], r2 = ts ? rS[o] : real(0.0);
        solve_row(P, g, k, kh[o], kh[o + n2], P.thv_dt_zero, R);
        R.r[0][k * SL_X] = r1;
        R.r[1][k * SL_X] = r2;
    }
    __syncthreads();
    solve_pairs(s_dyn, nz);
    __syncthreads();
#ifdef OC_MIXED
    const ColGeo64 g64 = ColGeo64::load(P, c);
#endif
#pragma unroll 2
    for (int k = first; k < nz; k += SL_Y) {
        const size_t o = (size_t)k * n2 + c;
        real m3;
        const real dz = g.dz(P, k, m3);
        const real Tn = R.r[0][k * SL_X] * m3;
        wide bn;
        if (ts) {
            const real Sn = R.r[1][k * SL_X] * m3;
#ifdef OC_MIXED
            const wide zc = g64.above(P, k) + 0.5 * g64.dz(P, k);
            (void)dz;
#else
            const wide zc = g.above(P, k) + real(0.5) * dz;
#endif
            bn = buoyancy_of(P, wide(Tn), wide(Sn), zc) * wide(m3);  // EOS in fp64 on both paths
            if (live) {
                T_out[o] = Tn;
                S_out[o] = Sn;
            }
        } else {
            bn = wide(Tn);
        }
        if (live) b_out[o] = bn;
    }
}

// diagnose b = EOS(T, S, zc) * m3 on the model grid (initial states)
__global__ void k_diag_buoyancy(KPR P, const real* __restrict__ T, const real* __restrict__ S,
                                wide* __restrict__ b) {
    COLUMN_PROLOGUE
    const size_t c = nb.c;
#ifdef OC_MIXED
    const ColGeo64 g64 = ColGeo64::load(P, (int)c);
    for (int k = 0; k < P.nz; ++k) {
        const size_t o = (size_t)k * n2 + c;
        const wide dz = g64.dz(P, k);
        const wide zc = g64.above(P, k) + 0.5 * dz;
        b[o] = buoyancy_of(P, wide(T[o]), wide(S[o]), zc) * (k < g64.kb ? 1.0 : 0.0);
    }
#else
    real above = real(0.0);
    for (int k = 0; k < P.nz; ++k) {
        const size_t o = (size_t)k * n2 + c;
        real m3;
        const real dz = col_dz(P, (int)c, k, m3);
        const real zc = above + real(0.5) * dz;
        above = (k == 0) ? dz : above + dz;
        b[o] = buoyancy_of(P, T[o], S[o], zc) * m3;
    }
#endif
}

// ------------------------------------------------------------------ transports
// depth-integrated transports sum_k dz3u u, sum_k dz3v v (fp64 sums on both paths), by
// levels on every grid: us a launch by columns and by levels, 128 x 4 x 32 5.1 and 1.5,
// 16,384 x 50 13 and 15, 262,144 x 50 113 and 49
__global__ void __launch_bounds__(LV_X * LV_Y) k_transport(KPR P, const real* __restrict__ u,
                                                           const real* __restrict__ v, wide* __restrict__ U,
                                                           wide* __restrict__ V) {
    __shared__ wide terms[2][LV_K][LV_X];
    LEVELS_PROLOGUE
    const size_t c = nb.c;
    const ColGeoR gc = ColGeoR::load(P, (int)c), ge = ColGeoR::load(P, nb.at(0, 1)), gn = ColGeoR::load(P, nb.at(1, 0));
    const int2 kf = P.kface[c];
    const int nz = P.nz;
    level_sums<2, false>(nz, terms, [&](int k, wide* t) {
        const size_t o = (size_t)k * n2 + c;
        real m;
        const real dzc = gc.dz(P, k, m);
        t[0] = wide(face_dz(P, kf.x, k, dzc, ge.dz(P, k, m)) * u[o]);
        t[1] = wide(face_dz(P, kf.y, k, dzc, gn.dz(P, k, m)) * v[o]);
    }, [&](int n, int k, wide sum) {
        if (k == nz - 1 && live) (n ? V : U)[c] = sum;
    });
}

// ------------------------------------------------------------------ launchers
#define NZ_DISPATCH(NZ, CALL)                \
    do {                                     \
        if ((NZ) + 1 <= 33) {                \
            constexpr int NZM = 33;          \
            CALL;                            \
        } else if ((NZ) + 1 <= 65) {         \
            constexpr int NZM = 65;          \
            CALL;                            \
        } else {                             \
            constexpr int NZM = OC_MAXNZ + 1; \
            CALL;                            \
        }                                    \
    } while (0)
void launch_qsolve(const KLR& P, const real* km, real* q, cudaStream_t s) {
    NZ_DISPATCH(P.nz, (k_qsolve<NZM><<<col_grid(P), col_block(), 0, s>>>(P, km, q)));
}
template <int NZM>
static void closure_nzm(const KLR& P, const real* u, const real* v, const wide* b, real* e, real* km, real* kh,
                        real* q, cudaStream_t s) {
    const dim3 blk = col_block();
#ifdef OC_MIXED
    const size_t smem = (size_t)(P.nz + 1) * blk.x * blk.y * sizeof(real);
    // above 48 KB a kernel's dynamic shared memory is opt-in, once per device
    static std::atomic<unsigned long long> opted{0};
    int dev = 0;
    cudaGetDevice(&dev);
    const unsigned long long bit = 1ULL << (dev & 63);
    if (!(opted.load() & bit)) {
        cudaFuncSetAttribute(k_closure<NZM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)((size_t)(NZM + 1) * blk.x * blk.y * sizeof(real)));
        opted.fetch_or(bit);
    }
#else
    const size_t smem = 0;
#endif
    k_closure<NZM><<<col_grid(P), blk, smem, s>>>(P, u, v, b, e, km, kh, q);
}
void launch_closure(const KLR& P, const real* u, const real* v, const wide* b, real* e,
                    real* km, real* kh, real* q, cudaStream_t s) {
    if (P.n2 <= closure_columns(P.nz)) {
        const size_t row = (size_t)5 * CL_X * sizeof(real);
        // above 48 KB a kernel's dynamic shared memory is opt-in, once per device
        static std::atomic<unsigned long long> opted{0};
        int dev = 0;
        cudaGetDevice(&dev);
        const unsigned long long bit = 1ULL << (dev & 63);
        if (!(opted.load() & bit)) {
            cudaFuncSetAttribute(k_closure_levels, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)((OC_MAXNZ + 1) * row));
            opted.fetch_or(bit);
        }
        const unsigned ctas = (unsigned)(((P.nx + CL_X - 1) / CL_X) * P.ny);
        k_closure_levels<<<ctas, dim3(CL_X, CL_Y), (P.nz + 1) * row, s>>>(P, u, v, b, e, km, kh, q);
        return;
    }
    NZ_DISPATCH(P.nz, (closure_nzm<NZM>(P, u, v, b, e, km, kh, q, s)));
}
void launch_kukv(const KPR& P, const real* q, wide* Ku, wide* Kv, cudaStream_t s) {
    if (P.n2 <= std::min(kFewColumns / 2, level_sum_columns(P.nz)))
        k_kukv_few<<<level_grid(P), level_block(), 0, s>>>(P, q, Ku, Kv);
    else
        k_kukv<<<col_grid(P), col_block(), 0, s>>>(P, q, Ku, Kv);
}
void launch_wcol(const KPR& P, const real* u, const real* v, real* w, cudaStream_t s) {
    if (P.n2 <= level_sum_columns(P.nz))
        k_wcol_few<<<level_grid(P), level_block(), 0, s>>>(P, u, v, w);
    else
        k_wcol<<<col_grid(P), col_block(), 0, s>>>(P, u, v, w);
}
void launch_phi(const KPR& P, const wide* b, wide* phi, cudaStream_t s) {
    k_phi<<<col_grid(P), col_block(), 0, s>>>(P, b, phi);
}
// Levels one CTA marches, for `tiles` tiles and `resident` CTAs on the GPU at once: the
// count whose rounds cost least, a round being its levels plus one (a CTA's start
// forms the fluxes at its top again and fills its pipeline). A small grid takes few
// levels, so that its tiles reach every SM; a large one takes what leaves the last
// round fullest. us a launch of k_mom_column and k_tracer_rhs with 10 levels on every
// grid and with these: 48 x 48 x 12 50 and 52, now 11 and 12; 128 x 4 x 32 25 and 33, now 5
// and 5; 512 x 512 x 50 1049 and 704, now 1043 and 691.
static int levels_per_cta(long long tiles, int nz, long long resident) {
    int best = nz;
    long long cost = -1;
    for (int slabs = 1; slabs <= nz; ++slabs) {
        const int kl = (nz + slabs - 1) / slabs;
        const long long rounds = (tiles * ((nz + kl - 1) / kl) + resident - 1) / resident;
        if (cost < 0 || rounds * (kl + 1) < cost) {
            cost = rounds * (kl + 1);
            best = kl;
        }
    }
    return best;
}
void default_levels(const KPR& P, int& mom_kl, int& tr_kl) {
    int dev = 0, sms = 1, m = 1, t = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, k_mom_column, MOM_TX * MOM_TY * 2, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&t, k_tracer_rhs, TRX * TRY, 0);
    const long long mt = (long long)((P.nx + MOM_TX - 1) / MOM_TX) * ((P.ny + MOM_TY - 1) / MOM_TY);
    const long long tt = (long long)((P.nx + TRX - 1) / TRX) * ((P.ny + TRY - 1) / TRY);
    mom_kl = levels_per_cta(mt, P.nz, (long long)sms * (m > 0 ? m : 1));
    tr_kl = levels_per_cta(tt, P.nz, (long long)sms * (t > 0 ? t : 1));
}
static dim3 cell_block() { return dim3(32, 8, 1); }
static dim3 cell_grid(const KPR& P) { return dim3((P.nx + 31) / 32, (P.ny + 7) / 8, P.nz); }
void launch_mom_explicit(const KLR& P, const real* u, const real* v, const wide* b,
                         const wide* phi, const real* w, const real* km, const wide* gx2, const wide* gy2,
                         real* pgx, real* pgy, real* avpv, real* avpu, real* dzu, real* dzv, real* stu, real* stv,
                         real* ru, real* rv, cudaStream_t s) {
    const dim3 grid((P.nx + MOM_TX - 1) / MOM_TX, (P.ny + MOM_TY - 1) / MOM_TY, (P.nz + P.mom_kl - 1) / P.mom_kl);
    k_mom_column<<<grid, dim3(MOM_TX, MOM_TY, 2), 0, s>>>(P, u, v, b, phi, w, km, gx2, gy2, pgx, pgy, avpv, avpu, dzu, dzv,
                                             stu, stv, ru, rv);
}
void launch_predictor_rhs(const KPR& P, const real* u, const real* v, const real* u_it,
                          const real* v_it, const real* pgx, const real* pgy, const real* avpv,
                          const real* avpu, const real* dzu, const real* dzv, const real* stu,
                          const real* stv, const wide* gx2, const wide* gy2, real* ru, real* rv,
                          cudaStream_t s) {
    k_predictor_rhs<<<cell_grid(P), cell_block(), 0, s>>>(P, u, v, u_it, v_it, pgx, pgy, avpv, avpu, dzu,
                                                          dzv, stu, stv, gx2, gy2, ru, rv);
}
void launch_momentum_solve(const KLR& P, const real* km, real* ghu, real* ghv, wide* Ug, wide* Vg,
                           cudaStream_t s) {
    if (P.n2 <= kFewColumns) {
        const dim3 grid((P.nx + 31) / 32, (P.ny + 1) / 2);
        NZ_DISPATCH(P.nz, (k_momentum_solve_few<NZM><<<grid, dim3(32, 2, 2), 0, s>>>(P, km, ghu, ghv, Ug, Vg)));
    } else {
        NZ_DISPATCH(P.nz, (k_momentum_solve<NZM><<<col_grid(P), col_block(), 0, s>>>(P, km, ghu, ghv, Ug, Vg)));
    }
}
void launch_backsub(const KPR& P, const real* ghu, const real* ghv, const real* q,
                    const wide* eta_new, real* u_out, real* v_out, cudaStream_t s) {
    if (P.n2 <= backsub_columns(P.nz))
        k_backsub_few<<<level_grid(P), level_block(), 0, s>>>(P, ghu, ghv, q, eta_new, u_out, v_out);
    else
        k_backsub<<<col_grid(P), col_block(), 0, s>>>(P, ghu, ghv, q, eta_new, u_out, v_out);
}
void launch_tracer_rhs(const KLR& P, const real* C0, const real* S, const real* u, const real* v,
                       const real* w, const real* kh, real* rT, real* rS, cudaStream_t s) {
    const dim3 grid((P.nx + TRX - 1) / TRX, (P.ny + TRY - 1) / TRY, (P.nz + P.tr_kl - 1) / P.tr_kl);
    k_tracer_rhs<<<grid, dim3(TRX, TRY), 0, s>>>(P, C0, S, u, v, w, kh, rT, rS);
}
void launch_tracer_solve(const KLR& P, const real* rT, const real* rS, const real* kh,
                         real* T_out, real* S_out, wide* b_out, cudaStream_t s) {
    if (P.n2 <= tracer_columns(P.nz)) {
        const size_t row = (size_t)5 * SL_X * sizeof(real);
        // above 48 KB a kernel's dynamic shared memory is opt-in, once per device
        static std::atomic<unsigned long long> opted{0};
        int dev = 0;
        cudaGetDevice(&dev);
        const unsigned long long bit = 1ULL << (dev & 63);
        if (!(opted.load() & bit)) {
            cudaFuncSetAttribute(k_tracer_levels, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(OC_MAXNZ * row));
            opted.fetch_or(bit);
        }
        const unsigned ctas = (unsigned)(((P.nx + SL_X - 1) / SL_X) * P.ny);
        k_tracer_levels<<<ctas, dim3(SL_X, SL_Y), P.nz * row, s>>>(P, rT, rS, kh, T_out, S_out, b_out);
        return;
    }
    NZ_DISPATCH(P.nz, (k_tracer_solve<NZM><<<col_grid(P), col_block(), 0, s>>>(P, rT, rS, kh, T_out,
                                                                             S_out, b_out)));
}
void launch_diag_buoyancy(const KPR& P, const real* T, const real* S, wide* b, cudaStream_t s) {
    k_diag_buoyancy<<<col_grid(P), col_block(), 0, s>>>(P, T, S, b);
}
void launch_transport(const KPR& P, const real* u, const real* v, wide* U, wide* V,
                      cudaStream_t s) {
    k_transport<<<level_grid(P), level_block(), 0, s>>>(P, u, v, U, V);
}

}  // namespace oc
