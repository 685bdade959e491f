// Shared by the Krylov translation units: scalar helpers, the BiCGStab state
// machine and the entry points one unit offers to another.
#pragma once

#include "gf_common.cuh"

namespace gf {

constexpr int kMaxBlocks = 1024;
constexpr int kMaxNV = 16;
constexpr int kCtlDoubles = 32;
constexpr long long kSpinLimit = 30000000LL;  // x ~40 ns polls: about a second

// Partial sums are double-buffered by barrier parity: a block may write the
// next barrier's partials while a slower block still reads this one's, but
// not the one after (that needs the slow block's arrival).
constexpr int64_t kPartials = 2LL * kMaxBlocks * kMaxNV;
constexpr int64_t kHeader = kCtlDoubles + kPartials;

struct KCtl {
    unsigned long long count;  // barrier arrivals since launch (zeroed per launch)
    int error;
    int pad;
};

__device__ __forceinline__ int vload(const int* p) { return *(const volatile int*)p; }

// Release-add / acquire-load pair of the grid barrier (the CTA barrier
// before the add makes it cumulative over the whole block's writes).
__device__ __forceinline__ void arrive_release(unsigned long long* p) {
    asm volatile("fence.acq_rel.gpu;\n\tred.relaxed.gpu.global.add.u64 [%0], 1;" ::"l"(p) : "memory");
}

__device__ __forceinline__ unsigned long long load_acquire(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// NaN: what a reduction that timed out has in place of its sums.
__device__ __forceinline__ double no_value() { return __longlong_as_double(0x7ff8000000000000LL); }

// Maximum that keeps a NaN (a norm with one must not pass a stopping test).
__device__ __forceinline__ double nmax(double a, double b) {
    if (a != a || b != b) return no_value();
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

// L2 prefetch of elements [c, c + cnt) of an array of n by one instruction
// (16-byte lines that hold at least one of them; nothing is read or faults).
__device__ __forceinline__ void pf_bulk(const void* base, int es, int c, int cnt, int n) {
    if (c >= n) return;
    const int end = n - c < cnt ? n : c + cnt;
    const uint64_t a0 = (reinterpret_cast<uint64_t>(base) + (uint64_t)c * es) & ~15ull;
    const uint64_t a1 = (reinterpret_cast<uint64_t>(base) + (uint64_t)end * es) & ~15ull;
    if (a1 > a0)
        asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a0), "r"((uint32_t)(a1 - a0)) : "memory");
}

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

// Grid BiCGStab kernels (gf_bicgstab.cu).
const void* bicgstab_kernel(const gf_krylov_t& k);
constexpr int kBicgThreads = 1024;

// Halo flags: one 64-bit epoch per block, one per 128-byte line (flags of
// neighbouring blocks sharing a line cost ~1.7 us an iteration at 262K
// cells), after z and the Jacobi inverse in the workspace.
constexpr int64_t kHaloFlagStride = 16;
constexpr int64_t kHaloFlagDoubles = kMaxBlocks * kHaloFlagStride;

// CG with the system resident on the grid's SMs (gf_resident.cu);
// GF_ERR_INVALID without a launch when it does not fit.
int launch_resident(const gf_krylov_t* k, cudaStream_t st);

// A solve on one thread-block cluster (gf_cluster.cu), for a system that
// cluster_fits.
bool cluster_fits(const gf_krylov_t& k, bool bicgstab);
int launch_cluster(const gf_krylov_t* k, bool bicgstab, cudaStream_t st);

}  // namespace gf
