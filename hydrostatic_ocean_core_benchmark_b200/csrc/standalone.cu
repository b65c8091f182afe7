// Standalone pieces of the step behind their own entry points, the B200 side of
// the reference's standalone kernel benches:
//   - the variable-coefficient free-surface Helmholtz solver on given face
//     coefficients (reference libs/cuda/src/helmholtz_bench.cu, solving the
//     system that tools/write_helmholtz_case.py writes with
//     libs/core/solvers_var.py HelmholtzVar) -> oc_helm_create / oc_helm_solve;
//   - the three equations of state on flat arrays (reference
//     libs/cuda/src/eos_bench.cu over libs/core/eos.py) -> oc_density.
// The solver is the step's own persistent cooperative HelmSolver, so its
// iteration counts and solutions are those of the step's solves; solver kind
// OC_SOLVER_PCG_REFINED selects the mixed-precision RefinedHelm instead.

#include <cuda_runtime.h>

#include <string>

#include "helm_refined.cuh"
#include "helmholtz.cuh"
#include "ocean_b200.h"
#include "oc_internal.cuh"

struct oc_helm {
    oc::HelmSolver solver;
    oc::RefinedHelm* refined = nullptr;  // set for OC_SOLVER_PCG_REFINED
    double* ku = nullptr;
    double* kv = nullptr;
    double* rhs = nullptr;  // device staging for host right-hand sides
    double* x = nullptr;
    int* status = nullptr;
    int nx = 0, ny = 0, device = 0;
    std::string err;
    ~oc_helm() {
        delete refined;
        for (void* p : {(void*)ku, (void*)kv, (void*)rhs, (void*)x, (void*)status})
            if (p) cudaFree(p);
    }
};

namespace {

int helm_fail(oc_helm* h, int code, const std::string& msg) {
    if (h) h->err = msg;
    return code;
}

// rho' for linear and S-EOS (eos.py:103-127), full in-situ rho for polyTEOS10-bsq
// (eos.py:68-100): what the reference's EOS bench evaluates per cell. A thread takes
// CELLS cells at a time, a block's width apart: their loads are all in flight before
// the first polynomial, and a coefficient fetched for one cell serves the others. Bound
// by fp64 issue (the polynomial is about 110 operations a cell): polyTEOS10 at 2e7 cells
// takes 208 us with one cell at a time and the kind tested inside, 189 with four. Where
// one cell per thread is at most two rounds of CTAs a call is bound by its latency instead, and
// a thread with four cells has four times the instructions to fetch and issue: a call of
// polyTEOS10 on 1,000 cells takes 14.2 us until its result with four, 11.8 with one, on
// 150,000 13.5 and 12.9 (among others 6.0 and 4.2, 4.5 and 4.2); on 320,000 7.2 and 6.2 among
// others, on 600,000 8.2 both.
template <int EOS>
__device__ __forceinline__ double density_of(double rho0, double alpha_t, double beta_s, double t0, double s0, double T,
                                             double S, double z) {
    return EOS == OC_EOS_TEOS10 ? oc::rho_teos10(T, S, z) : oc::rho_anomaly_of(EOS, rho0, alpha_t, beta_s, t0, s0, T, S, z);
}

template <int EOS, int CELLS>
__global__ void __launch_bounds__(256) k_density(double rho0, double alpha_t, double beta_s, double t0, double s0,
                                                 const double* __restrict__ T, const double* __restrict__ S,
                                                 const double* __restrict__ z, double* __restrict__ rho, int64_t n) {
    const int64_t tile = (int64_t)blockDim.x * CELLS;
    for (int64_t base = blockIdx.x * tile + threadIdx.x; base < n; base += gridDim.x * tile) {
        double Tv[CELLS], Sv[CELLS], zv[CELLS];
        if (base + (int64_t)(CELLS - 1) * blockDim.x < n) {
#pragma unroll
            for (int q = 0; q < CELLS; ++q) {
                const int64_t t = base + (int64_t)q * blockDim.x;
                Tv[q] = T[t];
                Sv[q] = S[t];
                zv[q] = z[t];
            }
#pragma unroll
            for (int q = 0; q < CELLS; ++q)
                rho[base + (int64_t)q * blockDim.x] = density_of<EOS>(rho0, alpha_t, beta_s, t0, s0, Tv[q], Sv[q], zv[q]);
        } else {
            for (int q = 0; q < CELLS; ++q) {
                const int64_t t = base + (int64_t)q * blockDim.x;
                if (t < n) rho[t] = density_of<EOS>(rho0, alpha_t, beta_s, t0, s0, T[t], S[t], z[t]);
            }
        }
    }
}

template <int EOS>
void density_launch(double rho0, double alpha_t, double beta_s, double t0, double s0, const double* T, const double* S,
                    const double* z, double* rho, int64_t count, cudaStream_t stream) {
    // CTAs that a B200's 148 SMs hold at once: eight an SM (five of polyTEOS10 with four cells). A
    // constant, as a query costs a small call more than it gives; on a part of a GPU the CTAs
    // only come in more rounds.
    constexpr int64_t block = 256, round = 148 * 8, cap = 4 * 148 * (EOS == OC_EOS_TEOS10 ? 5 : 8);
    if (count <= 2 * round * block) {
        k_density<EOS, 1><<<(unsigned)((count + block - 1) / block), block, 0, stream>>>(rho0, alpha_t, beta_s, t0, s0, T, S,
                                                                                    z, rho, count);
        return;
    }
    const int64_t need = (count + block * 4 - 1) / (block * 4);
    k_density<EOS, 4><<<(unsigned)(need < cap ? need : cap), block, 0, stream>>>(rho0, alpha_t, beta_s, t0, s0, T,
                                                                                        S, z, rho, count);
}

}  // namespace

extern "C" int oc_helm_create(const oc_helm_config* cfg, const double* ku, const double* kv,
                              const double* mask, oc_helm** out) {
    if (!cfg || !ku || !kv || !mask || !out) return OC_ERR_ARG;
    *out = nullptr;
    if (cfg->nx < 2 || cfg->ny < 2 || !(cfg->dx > 0.0) || !(cfg->dy > 0.0) || !(cfg->coef >= 0.0) ||
        !(cfg->rtol > 0.0) || cfg->max_iter < 1 || cfg->solver < OC_SOLVER_PCG_JACOBI ||
        cfg->solver > OC_SOLVER_PCG_MG)
        return OC_ERR_ARG;
    if (cudaSetDevice(cfg->device) != cudaSuccess) return OC_ERR_CUDA;
    oc_helm* h = new oc_helm();
    h->nx = cfg->nx;
    h->ny = cfg->ny;
    h->device = cfg->device;
    const size_t n = (size_t)cfg->nx * cfg->ny, bytes = n * sizeof(double);
    for (double** p : {&h->ku, &h->kv, &h->rhs, &h->x})
        if (cudaMalloc(p, bytes) != cudaSuccess) {
            delete h;
            return OC_ERR_CUDA;
        }
    if (cudaMalloc(&h->status, sizeof(int)) != cudaSuccess) {
        delete h;
        return OC_ERR_CUDA;
    }
    cudaMemset(h->status, 0, sizeof(int));
    cudaMemcpy(h->ku, ku, bytes, cudaMemcpyHostToDevice);
    cudaMemcpy(h->kv, kv, bytes, cudaMemcpyHostToDevice);
    if (cfg->solver == OC_SOLVER_PCG_REFINED) {
        h->refined = new oc::RefinedHelm();
        const int rc = h->refined->init(cfg->nx, cfg->ny, cfg->dx, cfg->dy, cfg->coef, cfg->rtol, cfg->max_iter,
                                        mask, h->ku, h->kv, h->err);
        if (rc) {
            delete h;
            return rc;
        }
    } else {
        const int rc = h->solver.init(cfg->nx, cfg->ny, cfg->dx, cfg->dy, cfg->coef, cfg->solver, cfg->rtol,
                                      cfg->max_iter, mask, h->ku, h->kv, 1, h->status, h->err);
        if (rc) {
            delete h;
            return rc;
        }
        h->solver.rebuild(0);
    }
    if (cudaDeviceSynchronize() != cudaSuccess) {
        delete h;
        return OC_ERR_CUDA;
    }
    *out = h;
    return OC_OK;
}

extern "C" int oc_helm_solve(oc_helm* h, const double* rhs, double* x, int32_t on_device,
                             int32_t* iterations, int32_t* converged, void* stream) {
    if (!h || !rhs || !x) return OC_ERR_ARG;
    cudaSetDevice(h->device);
    cudaStream_t s = (cudaStream_t)stream;
    const size_t bytes = (size_t)h->nx * h->ny * sizeof(double);
    const double* d_rhs = rhs;
    double* d_x = x;
    if (!on_device) {
        if (cudaMemcpyAsync(h->rhs, rhs, bytes, cudaMemcpyHostToDevice, s) != cudaSuccess)
            return helm_fail(h, OC_ERR_CUDA, "right-hand side upload failed");
        d_rhs = h->rhs;
        d_x = h->x;
    }
    int rc;
    if (h->refined) {
        rc = h->refined->solve(d_rhs, d_x, s, h->err);
    } else {
        cudaMemsetAsync(h->solver.d_log_count(), 0, sizeof(int), s);
        rc = h->solver.solve(d_rhs, d_x, s, h->err);
    }
    if (rc) return rc;
    if (!on_device && cudaMemcpyAsync(x, h->x, bytes, cudaMemcpyDeviceToHost, s) != cudaSuccess)
        return helm_fail(h, OC_ERR_CUDA, "solution download failed");
    const cudaError_t e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) return helm_fail(h, OC_ERR_CUDA, cudaGetErrorString(e));
    if (h->refined) return h->refined->report(iterations, converged, nullptr, nullptr, h->err);
    int st = 0, it = 0, cv = 0;
    cudaMemcpy(&st, h->status, sizeof(int), cudaMemcpyDeviceToHost);
    if (st) return helm_fail(h, st, "a device-side wait ran out its bound");
    cudaMemcpy(&it, h->solver.d_log_iters(), sizeof(int), cudaMemcpyDeviceToHost);
    cudaMemcpy(&cv, h->solver.d_log_conv(), sizeof(int), cudaMemcpyDeviceToHost);
    if (iterations) *iterations = it;
    if (converged) *converged = cv;
    return OC_OK;
}

extern "C" int oc_helm_refine_report(oc_helm* h, int32_t* refinement_steps, double* relative_residual) {
    if (!h) return OC_ERR_ARG;
    if (!h->refined) return helm_fail(h, OC_ERR_UNSUPPORTED, "not the refined solver");
    cudaSetDevice(h->device);
    int outer = 0;
    const int rc = h->refined->report(nullptr, nullptr, &outer, relative_residual, h->err);
    if (rc == OC_OK && refinement_steps) *refinement_steps = outer;
    return rc;
}

extern "C" int oc_helm_set_inner_rtol(oc_helm* h, double inner_rtol) {
    if (!h || !(inner_rtol > 0.0) || !(inner_rtol < 1.0)) return OC_ERR_ARG;
    if (!h->refined) return helm_fail(h, OC_ERR_UNSUPPORTED, "not the refined solver");
    h->refined->set_inner_rtol(inner_rtol);
    return OC_OK;
}

extern "C" const char* oc_helm_last_error(oc_helm* h) { return h ? h->err.c_str() : "null handle"; }

extern "C" int oc_helm_destroy(oc_helm* h) {
    if (!h) return OC_ERR_ARG;
    cudaSetDevice(h->device);
    delete h;
    return OC_OK;
}

extern "C" int oc_density(int32_t eos, double rho0, double alpha_t, double beta_s, double t0, double s0,
                          const double* T, const double* S, const double* z, double* rho, int64_t count,
                          void* stream) {
    if (!T || !S || !z || !rho || count < 0 || eos < OC_EOS_LINEAR || eos > OC_EOS_TEOS10) return OC_ERR_ARG;
    if (count == 0) return OC_OK;
    const cudaStream_t st = (cudaStream_t)stream;
    if (eos == OC_EOS_LINEAR) density_launch<OC_EOS_LINEAR>(rho0, alpha_t, beta_s, t0, s0, T, S, z, rho, count, st);
    else if (eos == OC_EOS_SEOS) density_launch<OC_EOS_SEOS>(rho0, alpha_t, beta_s, t0, s0, T, S, z, rho, count, st);
    else density_launch<OC_EOS_TEOS10>(rho0, alpha_t, beta_s, t0, s0, T, S, z, rho, count, st);
    return cudaGetLastError() == cudaSuccess ? OC_OK : OC_ERR_CUDA;
}
