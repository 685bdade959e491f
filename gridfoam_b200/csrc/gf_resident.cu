// Jacobi-PCG with the whole system resident on the grid's SMs (sm_100a).
//
// Beyond a cluster (gf_cluster.cu), up to 405,224 cells on 148 SMs (2,738 a
// block; octrees, with two further entries a cell, 311,688), a system's rows
// still fit the shared memory of all SMs together (80 bytes a cell: six
// coefficients, six neighbour codes and the block's own part of z) and its
// vectors their registers.  So an iteration touches global memory only for
// the z of other blocks' cells: the form it replaces at these sizes
// (pcg1_halo_body: r, p, q, w in shared memory, the rows read again every
// iteration) spent most of a pass on the chain length -> index -> gather
// through L2 and on 100 bytes a cell of L2 traffic.  Same arithmetic:
// Chronopoulos and Gear's one-reduction form with a halo sync between
// neighbouring blocks.
//
// Measured (us an iteration, the form before in brackets): boxes of 64K cells
// 5.5 (6.9), 115K 6.1 (7.1), 262K 7.6 (8.2), 389K 9.1 (9.5); octrees of 67K
// 6.3 (10.8), 236K 10.9 (14.7), 285K 12.5.  What bounds it: the reduction and
// the halo sync (3.3 us), then on octrees the blocks at level interfaces,
// which hold half as many entries again as the others.
#include "gf_gridsync.cuh"

namespace gf {

namespace {

constexpr int kRT = 512;
constexpr int kRSlots = 6;  // slots a cell in shared memory; longer rows keep the rest behind them
constexpr int kRSmemMax = 227 * 1024;

static size_t res_smem(int64_t chunk, size_t elem) {
    return (size_t)chunk * (elem + kRSlots * (elem + sizeof(int)));
}

using ResShared = GridShared<kRT, 3>;

// The entry of slot s of row c: neighbour and coefficient.  A box has
// implicit neighbours, and a symmetric one keeps its "-" coefficients in the
// "+" slots of the cells below.
__device__ __forceinline__ void row_entry(const gf_krylov_t& K, int c, int s, int& j, double& w) {
    const int n = (int)K.n;
    if (K.stride_y > 0) {
        const int st = s < 2 ? 1 : (s < 4 ? (int)K.stride_y : (int)K.stride_z);
        if (s & 1) {
            j = c < n - st ? c + st : c;
            w = __ldg(K.val + (int64_t)s * n + c);
        } else {
            j = c >= st ? c - st : c;
            w = !K.symmetric ? __ldg(K.val + (int64_t)s * n + c)
                             : (c >= st ? __ldg(K.val + (int64_t)(s + 1) * n + c - st) : 0.0);
        }
        return;
    }
    j = __ldg(K.nbr + (int64_t)s * n + c);
    w = __ldg(K.val + (int64_t)s * n + c);
}

// Publish epoch ep for this block, then wait (bounded) until blocks lo..hi
// have published it.
__device__ __forceinline__ bool res_halo(ResShared& sh, KCtl* ctl, unsigned long long* flags, unsigned long long ep,
                                         int lo, int hi) {
    __syncthreads();
    if (threadIdx.x == 0)
        asm volatile("fence.acq_rel.gpu;\n\tst.relaxed.gpu.global.u64 [%0], %1;" ::"l"(
                         flags + kHaloFlagStride * sh.bid),
                     "l"(ep)
                     : "memory");
    int err = 0;
    for (int b = lo + (int)threadIdx.x; b <= hi && !err; b += kRT) {
        if (b == sh.bid) continue;
        long long it = 0;
        while (load_acquire(flags + kHaloFlagStride * b) < ep) {
            __nanosleep(20);
            ++it;
            if ((it & 255) == 0 && vload(&ctl->error) != 0) {
                err = 1;
                break;
            }
            if (it > sh.spin) {
                atomicExch(&ctl->error, 1);
                err = 1;
                break;
            }
        }
    }
    return __syncthreads_or(err) == 0;
}

// WIDE: rows may be longer than six slots (cells with finer neighbours).  The
// further entries follow the six-slot arrays as far as there is room (extra
// entries), beyond that they are read from global memory.  (A table of the
// long rows worked off by all threads before the own cells was slower: 12.6
// against 10.9 us an iteration on the octree of 236K cells.)  On octrees the
// neighbouring blocks of a block span most of the grid, and the grid barrier
// is the faster halo sync (10.9 against 11.2 us).
template <int U, bool WIDE>
__global__ void __launch_bounds__(kRT, 1) k_pcg_resident(gf_krylov_t K, int chunk, int extra) {
    extern __shared__ __align__(16) char res_mem[];
    __shared__ ResShared sh;
    __shared__ int s_lo, s_hi, s_extra;
    KCtl* ctl = reinterpret_cast<KCtl*>(K.work);
    double* partials = K.work + kCtlDoubles;
    double* vec = partials + kPartials;
    const int n = (int)K.n, bid = (int)blockIdx.x;
    double* z = vec;
    unsigned long long* flags = reinterpret_cast<unsigned long long*>(vec + 2 * (int64_t)n);
    const int c0 = bid * chunk;
    const int m = n - c0 < chunk ? (n - c0 > 0 ? n - c0 : 0) : chunk;
    double* zs = reinterpret_cast<double*>(res_mem);
    double* val = zs + chunk;
    double* xval = val + (size_t)kRSlots * chunk;
    int* code = reinterpret_cast<int*>(xval + (WIDE ? extra : 0));
    int* xcode = code + (size_t)kRSlots * chunk;
    const bool jac = K.jacobi != 0, linf = K.norm_inf != 0;
    grid_init(sh, K, (int)gridDim.x, bid);
    if (threadIdx.x == 0) {
        s_lo = bid;
        s_hi = bid;
        s_extra = 0;
        flags[kHaloFlagStride * bid] = 0ull;  // seen by every block after the first reduction
    }
    __syncthreads();

    double x[U], r[U], p[U], q[U], w[U], iv[U], d[U];
    int len[U], at0[U];  // row lengths; places of the further entries (-1: global memory)
    // out[u]: the rows' products with the vector whose own part is `own` and
    // whose global values are `glob`; out holds the own cells' values.  A code
    // is the place in the block (>= 0) or ~cell; either way the value is one
    // generic load.
    auto value = [&](const double* own, const double* glob, int a) {
        const double* at = a >= 0 ? own + a : glob + ~a;
        return *at;
    };
    auto apply = [&](const double* own, const double* glob, double (&out)[U]) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = threadIdx.x + u * kRT;
            if (i >= m) continue;
            double acc = d[u] * out[u], g[kRSlots];
#pragma unroll
            for (int s = 0; s < kRSlots; ++s) g[s] = value(own, glob, code[s * chunk + i]);
#pragma unroll
            for (int s = 0; s < kRSlots; ++s) acc += val[s * chunk + i] * g[s];
            out[u] = acc;
        }
        if constexpr (WIDE) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int more = len[u] - kRSlots;
                for (int s0 = 0; s0 < more; s0 += 3) {
                    double a[3], g[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        a[k] = g[k] = 0.0;
                        if (s0 + k >= more) continue;
                        if (at0[u] >= 0) {
                            g[k] = value(own, glob, xcode[at0[u] + s0 + k]);
                            a[k] = xval[at0[u] + s0 + k];
                        } else {
                            int j;
                            row_entry(K, c0 + (int)threadIdx.x + u * kRT, kRSlots + s0 + k, j, a[k]);
                            g[k] = glob[j];
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 3; ++k)
                        if (s0 + k < more) out[u] += a[k] * g[k];
                }
            }
        }
    };
    double loc[2] = {0.0, 0.0};  // this thread's |r| and r.z of the last update
    int lo = bid, hi = bid;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int i = threadIdx.x + u * kRT, c = c0 + i;
        x[u] = r[u] = p[u] = q[u] = w[u] = iv[u] = d[u] = 0.0;
        len[u] = 0;
        at0[u] = -1;
        if (i >= m) continue;
        len[u] = K.stride_y > 0 || K.width == kRSlots ? kRSlots : (K.row_len ? (int)__ldg(K.row_len + c) : K.width);
        if (WIDE && len[u] > kRSlots) {
            at0[u] = atomicAdd(&s_extra, len[u] - kRSlots);
            if (at0[u] + len[u] - kRSlots > extra) at0[u] = -1;
        }
        for (int s = 0; s < len[u]; ++s) {
            int j;
            double a;
            row_entry(K, c, s, j, a);
            lo = j / chunk < lo ? j / chunk : lo;
            hi = j / chunk > hi ? j / chunk : hi;
            const int b = j >= c0 && j < c0 + m ? j - c0 : ~j;
            if (s < kRSlots) {
                val[s * chunk + i] = a;
                code[s * chunk + i] = b;
            } else if (at0[u] >= 0) {
                xval[at0[u] + s - kRSlots] = a;
                xcode[at0[u] + s - kRSlots] = b;
            }
        }
        for (int s = len[u]; s < kRSlots; ++s) {
            val[s * chunk + i] = 0.0;
            code[s * chunk + i] = i;
        }
        d[u] = __ldg(K.diag + c);
        iv[u] = inv_diag(K.diag, c, jac);
        w[u] = x[u] = K.x[c];
    }
    apply(K.x + c0, K.x, w);
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int i = threadIdx.x + u * kRT, c = c0 + i;
        if (i >= m) continue;
        r[u] = __ldg(K.rhs + c) - w[u];
        const double zk = iv[u] * r[u];
        zs[i] = zk;
        z[c] = zk;
        loc[0] = norm_acc(loc[0], r[u], linf);
        loc[1] += r[u] * zk;
    }
    atomicMin(&s_lo, lo);
    atomicMax(&s_hi, hi);
    bool ok = grid_sum<2>(sh, ctl, partials, loc, linf ? 1u : 0u);
    // (a wait that ran out leaves no totals)
    const double r0 = ok ? norm_fin(sh.total[0], linf) : no_value(), thresh = fmax(K.atol, K.rtol * r0);
    double fin = r0, rz = ok ? sh.total[1] : 0.0, alpha = 1.0;
    int its = 0, status = !ok ? -1 : (r0 < thresh ? GF_OK : (!isfinite(r0) ? GF_NONFINITE : -1));
    if (K.max_iter <= 0 && status < 0) status = GF_MAX_ITER;
    // Every thread holds the same scalars (from the same totals) and takes
    // the same branches.
    double rn = loc[0], gm = loc[1];
    for (int it = 1; ok && status < 0; ++it) {
        double sum[3] = {rn, gm, 0.0};
#pragma unroll
        for (int u = 0; u < U; ++u) w[u] = iv[u] * r[u];
        apply(zs, z, w);
#pragma unroll
        for (int u = 0; u < U; ++u) sum[2] += w[u] * (iv[u] * r[u]);
        ok = grid_sum<3>(sh, ctl, partials, sum, linf ? 1u : 0u);
        if (!ok) break;
        if (it > 1) {
            fin = norm_fin(sh.total[0], linf);
            its = it - 1;
            if (fin < thresh) status = GF_OK;
            else if (!isfinite(fin)) status = GF_NONFINITE;
            else if (its >= K.max_iter) status = GF_MAX_ITER;
            if (status >= 0) break;
        }
        const double g = it > 1 ? sh.total[1] : rz, beta = it > 1 ? g / rz : 0.0;
        alpha = g / (it > 1 ? sh.total[2] - beta * g / alpha : sh.total[2]);
        rz = g;
        rn = gm = 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = threadIdx.x + u * kRT;
            if (i >= m) continue;
            p[u] = iv[u] * r[u] + p[u] * beta;
            q[u] = w[u] + q[u] * beta;
            x[u] += alpha * p[u];
            r[u] -= alpha * q[u];
            const double zk = iv[u] * r[u];
            zs[i] = zk;
            z[c0 + i] = zk;
            rn = norm_acc(rn, r[u], linf);
            gm += r[u] * zk;
        }
        ok = WIDE ? grid_sync(sh, ctl) : res_halo(sh, ctl, flags, (unsigned long long)it, s_lo, s_hi);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int i = threadIdx.x + u * kRT;
        if (i < m) K.x[c0 + i] = x[u];
    }
    if (bid == 0 && threadIdx.x == 0) {
        double* o = K.stats;
        o[0] = r0;
        o[1] = fin;
        o[2] = its;
        o[3] = status == GF_OK;
        o[4] = ok ? (status < 0 ? GF_MAX_ITER : status) : GF_ERR_TIMEOUT;
    }
}

// The FP32-inner form: the updates of pcg1_mixed_halo_body (FP64 refinement
// around FP32 cycles, FP64 dot products, every cycle's true residual from the
// FP64 rows in global memory), with 52 bytes a cell on the SMs.
//
// Measured (us an inner iteration, the halo form in brackets): octrees of 41K
// cells 6.3 (8.7), 134K 8.3 (9.4), 236K 10.5 (14.5), 352K 13.4 (17.7); boxes of
// 34K 5.6 (6.5), 111K 6.3 (6.8), 262K 7.7 (7.9), but 524K 9.7 (9.0): a box's
// halo form reads no indices and its three or six coefficients are few bytes,
// so from more than four cells a thread on it is the faster.  1024 threads
// spill at 64 registers (6.2 at 34K, 10.8 at 524K).
template <int U, bool WIDE>
__global__ void __launch_bounds__(kRT, 1) k_pcg_mixed_resident(gf_krylov_t K, int chunk, int extra) {
    extern __shared__ __align__(16) char res_mem[];
    __shared__ ResShared sh;
    __shared__ int s_lo, s_hi, s_extra;
    KCtl* ctl = reinterpret_cast<KCtl*>(K.work);
    double* partials = K.work + kCtlDoubles;
    double* vec = partials + kPartials;
    const int n = (int)K.n, bid = (int)blockIdx.x;
    unsigned long long* flags = reinterpret_cast<unsigned long long*>(vec);
    float* z = reinterpret_cast<float*>(vec + n);
    const int c0 = bid * chunk;
    const int m = n - c0 < chunk ? (n - c0 > 0 ? n - c0 : 0) : chunk;
    float* zs = reinterpret_cast<float*>(res_mem);
    float* val = zs + chunk;
    float* xval = val + (size_t)kRSlots * chunk;
    int* code = reinterpret_cast<int*>(xval + (WIDE ? extra : 0));
    int* xcode = code + (size_t)kRSlots * chunk;
    const bool jac = K.jacobi != 0, linf = K.norm_inf != 0;
    grid_init(sh, K, (int)gridDim.x, bid);
    if (threadIdx.x == 0) {
        s_lo = bid;
        s_hi = bid;
        s_extra = 0;
        flags[kHaloFlagStride * bid] = 0ull;  // seen by every block after the first barrier
    }
    __syncthreads();

    float r[U], p[U], q[U], e[U], iv[U], d[U];  // e: the cycle's correction of x
    int len[U], at0[U];
    int lo = bid, hi = bid;
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int i = threadIdx.x + u * kRT, c = c0 + i;
        r[u] = p[u] = q[u] = e[u] = iv[u] = d[u] = 0.0f;
        len[u] = 0;
        at0[u] = -1;
        if (i >= m) continue;
        len[u] = K.stride_y > 0 || K.width == kRSlots ? kRSlots : (K.row_len ? (int)__ldg(K.row_len + c) : K.width);
        if (WIDE && len[u] > kRSlots) {
            at0[u] = atomicAdd(&s_extra, len[u] - kRSlots);
            if (at0[u] + len[u] - kRSlots > extra) at0[u] = -1;
        }
        for (int s = 0; s < len[u]; ++s) {
            int j;
            double a;
            row_entry(K, c, s, j, a);
            lo = j / chunk < lo ? j / chunk : lo;
            hi = j / chunk > hi ? j / chunk : hi;
            const int b = j >= c0 && j < c0 + m ? j - c0 : ~j;
            if (s < kRSlots) {
                val[s * chunk + i] = (float)a;
                code[s * chunk + i] = b;
            } else if (at0[u] >= 0) {
                xval[at0[u] + s - kRSlots] = (float)a;
                xcode[at0[u] + s - kRSlots] = b;
            }
        }
        for (int s = len[u]; s < kRSlots; ++s) {
            val[s * chunk + i] = 0.0f;
            code[s * chunk + i] = i;
        }
        d[u] = (float)__ldg(K.diag + c);
        iv[u] = (float)inv_diag(K.diag, c, jac);
    }
    atomicMin(&s_lo, lo);
    atomicMax(&s_hi, hi);

    auto value = [&](int a) {
        const float* at = a >= 0 ? zs + a : z + ~a;
        return *at;
    };
    auto row = [&](int u) {  // row u times z
        const int i = threadIdx.x + u * kRT;
        float acc = d[u] * (iv[u] * r[u]), g[kRSlots];
#pragma unroll
        for (int s = 0; s < kRSlots; ++s) g[s] = value(code[s * chunk + i]);
#pragma unroll
        for (int s = 0; s < kRSlots; ++s) acc += val[s * chunk + i] * g[s];
        return acc;
    };
    auto row_rest = [&](int u, float acc) {  // and its further entries
        const int more = len[u] - kRSlots;
        for (int s0 = 0; s0 < more; s0 += 3) {
            float a[3], g[3];
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                a[k] = g[k] = 0.0f;
                if (s0 + k >= more) continue;
                if (at0[u] >= 0) {
                    g[k] = value(xcode[at0[u] + s0 + k]);
                    a[k] = xval[at0[u] + s0 + k];
                } else {
                    int j;
                    double b;
                    row_entry(K, c0 + (int)threadIdx.x + u * kRT, kRSlots + s0 + k, j, b);
                    g[k] = z[j];
                    a[k] = (float)b;
                }
            }
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (s0 + k < more) acc += a[k] * g[k];
        }
        return acc;
    };
    // Every thread holds the same scalars (from the same totals) and takes
    // the same branches.
    bool ok = true, pending = false;
    int its = 0, status = -1;
    double r0 = 0.0, fin = 0.0, thresh = 0.0, rz = 0.0, alpha = 1.0, target = 0.0;
    unsigned long long ep = 0;
    for (int cycle = 0; ok && cycle <= K.max_outer; ++cycle) {
        // fold the correction, then the true residual in FP64
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = threadIdx.x + u * kRT;
            if (pending && i < m) K.x[c0 + i] += (double)e[u];
        }
        pending = false;
        ok = grid_sync(sh, ctl);
        if (!ok) break;
        double loc[2] = {0.0, 0.0};
#pragma unroll 1
        for (int u = 0; u < U; ++u) {
            const int i = threadIdx.x + u * kRT, c = c0 + i;
            if (i >= m) continue;
            double acc = __ldg(K.diag + c) * __ldcg(K.x + c);
            const int ln = K.stride_y > 0 || K.width == kRSlots ? kRSlots : (K.row_len ? (int)__ldg(K.row_len + c) : K.width);
            for (int s = 0; s < ln; ++s) {
                int j;
                double a;
                row_entry(K, c, s, j, a);
                acc += a * __ldcg(K.x + j);
            }
            const double rk = __ldg(K.rhs + c) - acc;
            loc[0] = norm_acc(loc[0], rk, linf);
            zs[i] = (float)rk;  // into registers below (u is no constant here)
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = threadIdx.x + u * kRT;
            if (i >= m) continue;
            r[u] = zs[i];
            e[u] = p[u] = q[u] = 0.0f;
            const float zk = iv[u] * r[u];
            zs[i] = zk;
            z[c0 + i] = zk;
            loc[1] += (double)r[u] * (double)zk;
        }
        ok = grid_sum<2>(sh, ctl, partials, loc, linf ? 1u : 0u);
        if (!ok) break;
        fin = norm_fin(sh.total[0], linf);
        if (cycle == 0) {
            r0 = fin;
            thresh = fmax(K.atol, K.rtol * fin);
        }
        if (fin < thresh) status = GF_OK;
        else if (!isfinite(fin)) status = GF_NONFINITE;
        if (status >= 0 || cycle == K.max_outer || its >= K.max_iter) break;
        rz = sh.total[1];
        alpha = 1.0;
        target = fmax(K.inner_eta * fin, (K.inner_margin > 0.0 ? K.inner_margin : 0.5) * thresh);
        pending = true;
        double rn = 0.0, gm = 0.0;  // this thread's |r| and r.z of the last update
        for (int k = 1;; ++k) {
            double sum[3] = {rn, gm, 0.0};
            float w[U];
#pragma unroll
            for (int u = 0; u < U; ++u) w[u] = (int)threadIdx.x + u * kRT < m ? row(u) : 0.0f;
            if constexpr (WIDE)
#pragma unroll
                for (int u = 0; u < U; ++u) w[u] = row_rest(u, w[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) sum[2] += (double)w[u] * (double)(iv[u] * r[u]);
            ok = grid_sum<3>(sh, ctl, partials, sum, linf ? 1u : 0u);
            if (!ok) break;
            if (k > 1) {
                const double nr = norm_fin(sh.total[0], linf);
                if (!(nr >= target) || !isfinite(nr)) break;
            }
            if (its >= K.max_iter) break;
            const double g = k > 1 ? sh.total[1] : rz, b = k > 1 ? g / rz : 0.0;
            alpha = g / (k > 1 ? sh.total[2] - b * g / alpha : sh.total[2]);
            rz = g;
            ++its;
            const float al = (float)alpha, be = (float)b;
            rn = gm = 0.0;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int i = threadIdx.x + u * kRT;
                if (i >= m) continue;
                p[u] = iv[u] * r[u] + p[u] * be;
                q[u] = w[u] + q[u] * be;
                e[u] += al * p[u];
                r[u] -= al * q[u];
                const float zk = iv[u] * r[u];
                zs[i] = zk;
                z[c0 + i] = zk;
                rn = norm_acc(rn, (double)r[u], linf);
                gm += (double)r[u] * (double)zk;
            }
            ++ep;
            ok = WIDE ? grid_sync(sh, ctl) : res_halo(sh, ctl, flags, ep, s_lo, s_hi);
            if (!ok) break;
        }
    }
    if (bid == 0 && threadIdx.x == 0) {
        double* o = K.stats;
        o[0] = r0;
        o[1] = fin;
        o[2] = its;
        o[3] = status == GF_OK;
        o[4] = ok ? (status < 0 ? GF_MAX_ITER : status) : GF_ERR_TIMEOUT;
    }
}

template <bool WIDE>
static const void* res_kernel(int u) {
    return u <= 1 ? (const void*)k_pcg_resident<1, WIDE>
                  : (u <= 2 ? (const void*)k_pcg_resident<2, WIDE>
                            : (u <= 4 ? (const void*)k_pcg_resident<4, WIDE> : (const void*)k_pcg_resident<6, WIDE>));
}

template <bool WIDE>
static const void* res_mixed_kernel(int u) {
    return u <= 1 ? (const void*)k_pcg_mixed_resident<1, WIDE>
                  : (u <= 2 ? (const void*)k_pcg_mixed_resident<2, WIDE>
                            : (u <= 4 || !WIDE ? (const void*)k_pcg_mixed_resident<4, WIDE>
                                               : (const void*)k_pcg_mixed_resident<6, true>));
}

}  // namespace

int launch_resident(const gf_krylov_t* k, cudaStream_t st) {
    // FP64: z, the (unused) inverse's place and the halo flags of the halo
    // form's workspace.  FP32-inner: the flags in the n doubles before z.
    const bool mixed = k->mixed != 0;
    const size_t elem = mixed ? sizeof(float) : sizeof(double);
    if (mixed ? k->n < kHaloFlagDoubles : k->work_len < kHeader + 2 * k->n + kHaloFlagDoubles) return GF_ERR_INVALID;
    // int indices of slot x n
    if ((int64_t)(k->width > 6 ? k->width : 6) * k->n >= (1LL << 31) || k->width < kRSlots) return GF_ERR_INVALID;
    int dev = 0, sms = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) {
        set_error("gf_pcg_solve: %s", cudaGetErrorString(e));
        return GF_ERR_CUDA;
    }
    const bool wide = k->width > kRSlots;
    int64_t grid = (k->n + kRT - 1) / kRT;
    if (grid > sms) grid = sms;
    if (k->block_cap > 0 && grid > k->block_cap) grid = k->block_cap;
    const int64_t chunk = (k->n + grid - 1) / grid;
    size_t smem = res_smem(chunk, elem);
    const int u = (int)((chunk + kRT - 1) / kRT);
    const size_t room = (size_t)kRSmemMax - sizeof(ResShared) - 1024;
    // FP32-inner: boxes of four and octrees of five cells a thread are the
    // largest that were measured to gain (262K and 352K cells).
    if (u > (!mixed ? 6 : (wide ? 5 : 4)) || smem > room) return GF_ERR_INVALID;
    // Further entries: what is left of the room.  With less than two a cell
    // the blocks at a level interface run out of it and the q-recurrence form
    // is the faster (octree of 349K cells with 1.1 a cell: 20 against 16 us
    // an iteration; 285K with 2.8: 12.5 against 13.7).
    int extra = 0;
    if (k->width > kRSlots) {
        const size_t kEntry = elem + sizeof(int);
        if (smem + 2 * chunk * kEntry > room) return GF_ERR_INVALID;
        const int64_t fit = (int64_t)((room - smem) / kEntry) & ~1LL, all = (chunk * (k->width - kRSlots) + 1) & ~1LL;
        extra = (int)(fit < all ? fit : all);
        smem += extra * kEntry;
    }
    grid = (k->n + chunk - 1) / chunk;
    const void* kern = mixed ? (wide ? res_mixed_kernel<true>(u) : res_mixed_kernel<false>(u))
                             : (wide ? res_kernel<true>(u) : res_kernel<false>(u));
    int occ = 0;
    // The attribute is the kernel's, not the launch's: set to the same bound by
    // every caller, or a thread with a smaller system would take it below what
    // another is about to launch with.
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, kRT, smem);
    if (e == cudaSuccess && (int64_t)occ * sms < grid) return GF_ERR_INVALID;
    if (e == cudaSuccess) e = cudaMemsetAsync(k->work, 0, sizeof(KCtl), st);
    gf_krylov_t arg = *k;
    int carg = (int)chunk;
    void* args[] = {&arg, &carg, &extra};
    if (e == cudaSuccess) e = cudaLaunchCooperativeKernel(kern, dim3((unsigned)grid), dim3(kRT), args, smem, st);
    if (e != cudaSuccess) {
        set_error("gf_pcg_solve: resident CG launch failed: %s", cudaGetErrorString(e));
        return GF_ERR_CUDA;
    }
    return GF_OK;
}

}  // namespace gf
