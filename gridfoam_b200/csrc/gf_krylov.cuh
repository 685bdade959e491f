// Shared by the Krylov translation units: scalar helpers, the BiCGStab state
// machine and the entry points one unit offers to another.
#pragma once

#include "gf_common.cuh"

namespace gf {

constexpr int kMaxBatch = 16;  // systems of a batched launch

// Maximum that keeps a NaN (a norm with one must not pass a stopping test).
__device__ __forceinline__ double nmax(double a, double b) {
    if (a != a || b != b) return __longlong_as_double(0x7ff8000000000000LL);
    return fmax(a, b);
}

__device__ __forceinline__ double comb(double x, double y, bool mx) { return mx ? nmax(x, y) : x + y; }

__device__ __forceinline__ double inv_diag(const double* __restrict__ diag, int64_t c, bool jac) {
    if (!jac) return 1.0;
    const double d = __ldg(diag + c);
    return fabs(d) < 2.220446049250313e-16 ? 1.0 : 1.0 / d;
}

__device__ __forceinline__ double norm_acc(double acc, double r, bool linf) {
    return linf ? nmax(acc, fabs(r)) : acc + r * r;
}

__device__ __forceinline__ double norm_fin(double acc, bool linf) { return linf ? acc : sqrt(acc); }

// BiCGStab per-component modes.
enum { kDone = 0, kRun = 1, kRestart = 2, kIdle = 3, kConvS = 4 };

struct BiState {
    double thresh, r0, final, rho_old, alpha, omega, beta;
    int mode, restarts, its, converged, status;
};

__device__ __forceinline__ void breakdown(BiState& s, int it, int max_restart) {
    if (s.restarts >= max_restart) {
        s.mode = kDone;
        s.its = it;
        s.status = GF_BREAKDOWN;
    } else {
        s.restarts += 1;
        s.mode = kRestart;
    }
}

// Solves on one thread-block cluster a system (gf_cluster.cu).  The launch
// functions return GF_ERR_INVALID without a launch when a system does not
// qualify; cluster_fits says so beforehand.
bool cluster_fits(const gf_krylov_t& k, bool bicgstab);
int launch_cluster(const gf_krylov_t* sys, int count, bool bicgstab, bool batched, cudaStream_t st);

}  // namespace gf
