// FP64 BiCGStab on the whole grid (sm_100a): one persistent cooperative
// launch for up to three components that share the matrix reads, for systems
// beyond what a cluster holds (gf_cluster.cu) and for callers that bound the
// blocks or the waits.  (The batched form, which gives each system a share of
// the blocks, is in gf_krylov.cu.)
//
// The reference's right-preconditioned BiCGStab (bicgstab.py:76-272), its
// breakdown tests and restarts included, in five passes over the cells:
//   P1  v = A M p              sums r_hat.v, |v|^2
//   P2  s = r - alpha v
//   P3  t = A M s              sums |s|, t.t, t.s
//   P4  x += alpha M p + omega M s, r = s - omega t    sums |r|, r_hat.r
//   P5  p = r + beta (p - omega v)
// What bounds it: at 1e5 cells the synchronisation, beyond L2 the bytes (640
// a cell and iteration for three components).  So the passes are ordered for
// few and cheap synchronisations: three reductions and two bare barriers an
// iteration (|s| is summed with t's values, |r_hat|^2 changes only at a
// restart and is kept), a reduction goes through shared memory with one warp
// a value instead of a shuffle tree a value in every warp, and the scalar
// updates of the components run on one thread each.  1024 threads at 64
// registers and cells taken in grid stride: 512 threads at 128 registers on
// contiguous chunks were slower at every size (4M-cell octree: 1138 us an
// iteration against 610; 147K-cell box: 32.8 against 29.8).
//
// Measured (three components, us an iteration, the form with five full
// reductions of up to twelve values before it in brackets): 25.7 (57) on a
// box of 147K cells, 80 (179) at 535K, 44 (80) on an octree of 236K, 265 at
// 1.73M, 605 (1000) at 4.08M: 4.3 TB/s of the 640 bytes a cell.
#include "gf_gridsync.cuh"

namespace gf {

namespace {

constexpr int kT = kBicgThreads;
// Row forms: any ELL rows, rows of exactly six slots, and six slots with the
// implicit neighbours of a uniform lexicographic box (the index table is not
// read, and the gathers do not wait for it).
enum { kEll = 0, kEll6 = 1, kBox = 2 };

struct BiShared : GridShared<kT, 9> {
    double hh[3];  // |r_hat|^2
    int restart;
};

// out_k = diag g(k, c) + sum_s val(s, c) g(k, nbr(s, c)), the loads of GRP
// slots issued before their products.
template <int NC, int ROWS, int GRP, class G>
__device__ __forceinline__ void bi_row(const gf_krylov_t& K, int c, const G& g, double (&out)[NC]) {
    static_assert(6 % GRP == 0, "six-slot rows are read in whole groups");
    const int n = (int)K.n;
    const double d = __ldg(K.diag + c);
#pragma unroll
    for (int k = 0; k < NC; ++k) out[k] = d * g(k, c);
    const int W = ROWS != kEll ? 6 : (K.row_len ? (int)__ldg(K.row_len + c) : K.width);
#pragma unroll
    for (int s0 = 0; s0 < W; s0 += GRP) {
        int nb[GRP];
        double a[GRP];
#pragma unroll
        for (int j = 0; j < GRP; ++j) {
            const int s = s0 + j;
            const bool in = ROWS != kEll || s < W;
            if constexpr (ROWS == kBox) {
                // the coefficient of a boundary slot is zero, so a wrapped or
                // clamped neighbour is harmless
                const int st = s < 2 ? 1 : (s < 4 ? (int)K.stride_y : (int)K.stride_z);
                nb[j] = (s & 1) ? (c < n - st ? c + st : c) : (c >= st ? c - st : c);
            } else {
                nb[j] = in ? __ldg(K.nbr + s * n + c) : c;
            }
            a[j] = in ? __ldg(K.val + s * n + c) : 0.0;
        }
#pragma unroll
        for (int j = 0; j < GRP; ++j)
            if (ROWS != kEll || s0 + j < W)
#pragma unroll
                for (int k = 0; k < NC; ++k) out[k] += a[j] * g(k, nb[j]);
    }
}

template <int NC, int ROWS>
__device__ __forceinline__ void bicgstab_body(const gf_krylov_t& K, int bk, int nbk, BiShared& sh, BiState* st) {
    // Six slots of three components at once spill at 64 registers (4M-cell
    // octree: 595 us an iteration against 609, but 96.6 against 90.5 at 535K
    // cells of a box); two at a time: 657.
    constexpr int GRP = NC > 1 ? 3 : 6;
    KCtl* ctl = reinterpret_cast<KCtl*>(K.work);
    grid_init(sh, K, nbk, bk);
    __syncthreads();
    double* partials = K.work + kCtlDoubles;
    double* vec = partials + kPartials;
    const int64_t n = K.n;
    double* r = vec;
    double* rh = vec + NC * n;
    double* p = vec + 2 * NC * n;
    double* v = vec + 3 * NC * n;
    double* s = vec + 4 * NC * n;
    double* t = vec + 5 * NC * n;
    double* inv = vec + 6 * NC * n;
    double* x = K.x;
    const bool jac = K.jacobi != 0, linf = K.norm_inf != 0;
    const unsigned nmask = linf ? ((1u << NC) - 1u) : 0u;
    const int c0 = bk * kT + (int)threadIdx.x, c1 = (int)n, step = nbk * kT;
    const int me = (int)threadIdx.x;  // < NC: the component whose scalars this thread updates
    bool ok;

    {  // r = b - A x; r_hat = p = r; |r|, r.r; the Jacobi inverse
        double loc[2 * NC];
#pragma unroll
        for (int j = 0; j < 2 * NC; ++j) loc[j] = 0.0;
        auto gx = [&](int k, int i) { return x[k * n + i]; };
        for (int c = c0; c < c1; c += step) {
            inv[c] = inv_diag(K.diag, c, jac);
            double ax[NC];
            bi_row<NC, ROWS, GRP>(K, c, gx, ax);
#pragma unroll
            for (int k = 0; k < NC; ++k) {
                const double rk = __ldg(K.rhs + k * n + c) - ax[k];
                r[k * n + c] = rk;
                rh[k * n + c] = rk;
                p[k * n + c] = rk;
                loc[k] = norm_acc(loc[k], rk, linf);
                loc[NC + k] += rk * rk;
            }
        }
        ok = grid_sum<2 * NC>(sh, ctl, partials, loc, nmask);
        if (me < NC) {
            BiState& b = st[me];
            // a wait that ran out leaves no totals
            const double r0 = ok ? norm_fin(sh.total[me], linf) : no_value();
            b.r0 = r0;
            b.final = r0;
            b.thresh = fmax(K.atol, K.rtol * r0);
            b.rho_old = sh.hh[me] = ok ? sh.total[NC + me] : 0.0;
            b.restarts = 0;
            b.its = 0;
            b.converged = 0;
            b.status = GF_MAX_ITER;
            b.mode = kRun;
            b.alpha = b.omega = b.beta = 0.0;
            if (r0 < b.thresh) {
                b.mode = kDone;
                b.converged = 1;
                b.status = GF_OK;
            } else if (!isfinite(r0)) {
                b.mode = kDone;
                b.status = GF_NONFINITE;
            }
        }
        __syncthreads();
    }
    // A restarting component takes r_hat = p = r in the pass after its
    // breakdown and idles for the rest of the iteration.
    auto copy_r = [&](int k, int c) {
        const double rk = r[k * n + c];
        rh[k * n + c] = rk;
        p[k * n + c] = rk;
        return rk * rk;
    };
    auto restarted = [&](int j) {
        st[me].rho_old = sh.hh[me] = sh.total[j];
        st[me].mode = kIdle;
    };

    for (int it = 1; ok && it <= K.max_iter; ++it) {
        int run = 0;
        if (me < NC) {
            if (st[me].mode == kIdle) st[me].mode = kRun;
            run = st[me].mode == kRun;
        }
        if (!__syncthreads_or(run)) break;

        {  // P1
            double loc[2 * NC];
#pragma unroll
            for (int j = 0; j < 2 * NC; ++j) loc[j] = 0.0;
            auto gy = [&](int k, int i) { return inv[i] * p[k * n + i]; };
            for (int c = c0; c < c1; c += step) {
                double av[NC];
                bi_row<NC, ROWS, GRP>(K, c, gy, av);
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    if (st[k].mode != kRun) continue;
                    v[k * n + c] = av[k];
                    loc[k] += rh[k * n + c] * av[k];
                    loc[NC + k] += av[k] * av[k];
                }
            }
            ok = grid_sum<2 * NC>(sh, ctl, partials, loc, 0u);
            if (!ok) break;
            if (me < NC && st[me].mode == kRun) {
                BiState& b = st[me];
                const double da = sh.total[me];
                if (fabs(da) <= 1e-6 * sqrt(sh.hh[me]) * sqrt(sh.total[NC + me])) breakdown(b, it, K.max_restart);
                else b.alpha = b.rho_old / da;
            }
            __syncthreads();
        }
        // P2
        for (int c = c0; c < c1; c += step)
#pragma unroll
            for (int k = 0; k < NC; ++k)
                if (st[k].mode == kRun) s[k * n + c] = r[k * n + c] - st[k].alpha * v[k * n + c];
        ok = grid_sync(sh, ctl);
        if (!ok) break;
        {  // P3 (and the restarts of P1's breakdowns)
            double loc[3 * NC];
#pragma unroll
            for (int j = 0; j < 3 * NC; ++j) loc[j] = 0.0;
            auto gz = [&](int k, int i) { return inv[i] * s[k * n + i]; };
            for (int c = c0; c < c1; c += step) {
                double at[NC];
                bi_row<NC, ROWS, GRP>(K, c, gz, at);
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    const int md = st[k].mode;
                    if (md == kRun) {
                        const double sk = s[k * n + c];
                        t[k * n + c] = at[k];
                        loc[k] = norm_acc(loc[k], sk, linf);
                        loc[NC + k] += at[k] * at[k];
                        loc[2 * NC + k] += at[k] * sk;
                    } else if (md == kRestart) {
                        loc[NC + k] += copy_r(k, c);
                    }
                }
            }
            ok = grid_sum<3 * NC>(sh, ctl, partials, loc, nmask);
            if (!ok) break;
            if (me < NC) {
                BiState& b = st[me];
                if (b.mode == kRestart) {
                    restarted(NC + me);
                } else if (b.mode == kRun) {
                    const double fin = norm_fin(sh.total[me], linf);
                    b.final = fin;
                    if (fin < b.thresh) {
                        b.mode = kConvS;
                        b.converged = 1;
                        b.its = it;
                        b.status = GF_OK;
                    } else if (!isfinite(fin)) {
                        b.mode = kDone;
                        b.its = it;
                        b.status = GF_NONFINITE;
                    } else {
                        const double dd = sh.total[NC + me], tn = sqrt(dd);
                        if (fabs(dd) <= 1e-6 * tn * tn) {
                            breakdown(b, it, K.max_restart);
                        } else {
                            b.omega = sh.total[2 * NC + me] / dd;
                            if (fabs(b.omega) <= 1e-6) breakdown(b, it, K.max_restart);
                        }
                    }
                }
            }
            __syncthreads();
        }
        {  // P4 (converged-on-s components take x += alpha y; P3's restarts)
            double loc[3 * NC];
#pragma unroll
            for (int j = 0; j < 3 * NC; ++j) loc[j] = 0.0;
            for (int c = c0; c < c1; c += step) {
                const double ic = inv[c];
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    const int md = st[k].mode;
                    if (md == kRun) {
                        const double sk = s[k * n + c];
                        const double y = ic * p[k * n + c];
                        const double z = ic * sk;
                        x[k * n + c] = x[k * n + c] + st[k].alpha * y + st[k].omega * z;
                        const double rk = sk - st[k].omega * t[k * n + c];
                        r[k * n + c] = rk;
                        loc[k] = norm_acc(loc[k], rk, linf);
                        loc[NC + k] += rh[k * n + c] * rk;
                        if (linf) loc[2 * NC + k] += rk * rk;
                    } else if (md == kConvS) {
                        x[k * n + c] = x[k * n + c] + st[k].alpha * (ic * p[k * n + c]);
                    } else if (md == kRestart) {
                        loc[NC + k] += copy_r(k, c);
                    }
                }
            }
            if (linf) {
                ok = grid_sum<3 * NC>(sh, ctl, partials, loc, nmask);
            } else {  // the 2-norm's own sum is |r|^2
                double two[2 * NC];
#pragma unroll
                for (int j = 0; j < 2 * NC; ++j) two[j] = loc[j];
                ok = grid_sum<2 * NC>(sh, ctl, partials, two, 0u);
            }
            if (!ok) break;
            if (threadIdx.x == 0) sh.restart = 0;
            __syncwarp();
            if (me < NC) {
                BiState& b = st[me];
                if (b.mode == kConvS) {
                    b.mode = kDone;
                } else if (b.mode == kRestart) {
                    restarted(NC + me);
                } else if (b.mode == kRun) {
                    const double fin = norm_fin(sh.total[me], linf);
                    const double rr = linf ? sh.total[2 * NC + me] : sh.total[me];
                    b.final = fin;
                    if (fin < b.thresh) {
                        b.mode = kDone;
                        b.converged = 1;
                        b.its = it;
                        b.status = GF_OK;
                    } else if (!isfinite(fin)) {
                        b.mode = kDone;
                        b.its = it;
                        b.status = GF_NONFINITE;
                    } else {
                        const double rho_new = sh.total[NC + me];
                        if (fabs(rho_new) <= 1e-6 * sqrt(sh.hh[me]) * sqrt(rr)) {
                            breakdown(b, it, K.max_restart);
                            if (b.mode == kRestart) sh.restart = 1;
                        } else {
                            b.beta = (rho_new / b.rho_old) * (b.alpha / b.omega);
                            b.rho_old = rho_new;
                        }
                    }
                }
            }
            __syncthreads();
        }
        {  // P5 (and the restarts of P4's breakdowns)
            double loc[NC];
#pragma unroll
            for (int k = 0; k < NC; ++k) loc[k] = 0.0;
            for (int c = c0; c < c1; c += step) {
#pragma unroll
                for (int k = 0; k < NC; ++k) {
                    const int md = st[k].mode;
                    if (md == kRun)
                        p[k * n + c] = r[k * n + c] + st[k].beta * (p[k * n + c] - st[k].omega * v[k * n + c]);
                    else if (md == kRestart)
                        loc[k] += copy_r(k, c);
                }
            }
            if (sh.restart) {
                ok = grid_sum<NC>(sh, ctl, partials, loc, 0u);
                if (!ok) break;
                if (me < NC && st[me].mode == kRestart) restarted(me);
            } else {
                ok = grid_sync(sh, ctl);
            }
            __syncthreads();
        }
    }
    if (bk == 0 && threadIdx.x == 0) {
        for (int k = 0; k < NC; ++k) {
            double* o = K.stats + 5 * k;
            const bool fin = st[k].mode == kDone;
            o[0] = st[k].r0;
            o[1] = st[k].final;
            o[2] = fin ? st[k].its : K.max_iter;
            o[3] = st[k].converged;
            o[4] = ok ? (fin ? st[k].status : GF_MAX_ITER) : GF_ERR_TIMEOUT;
        }
    }
}

// The shared memory is declared in the kernels: declared in a function that
// the linker sees called, it would count against every kernel of the library.
template <int NC, int ROWS>
__global__ void __launch_bounds__(kT, 1) k_bicgstab(gf_krylov_t K) {
    __shared__ BiShared sh;
    __shared__ BiState st[NC];
    bicgstab_body<NC, ROWS>(K, (int)blockIdx.x, (int)gridDim.x, sh, st);
}

}  // namespace

template <int ROWS>
static const void* bi_kernel(int ncomp) {
    return ncomp == 1 ? (const void*)k_bicgstab<1, ROWS>
                      : (ncomp == 2 ? (const void*)k_bicgstab<2, ROWS> : (const void*)k_bicgstab<3, ROWS>);
}

const void* bicgstab_kernel(const gf_krylov_t& k) {
    return k.stride_y > 0 ? bi_kernel<kBox>(k.ncomp) : (k.width == 6 ? bi_kernel<kEll6>(k.ncomp) : bi_kernel<kEll>(k.ncomp));
}

}  // namespace gf
