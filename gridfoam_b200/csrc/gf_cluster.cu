// Krylov solves of small systems on one thread-block cluster each (sm_100a).
//
// A system of a few ten thousand cells is bound by the synchronisation of
// its dot products, not by arithmetic or bandwidth: with the persistent
// grid kernels a Jacobi-PCG iteration of 8K to 33K cells takes 6.4-6.7 us
// and a three-component BiCGStab iteration 42 us, nearly all of it in grid
// reductions through L2 (2-3 us each).  Here the whole system lives on the
// chip: a cluster of up to 16 blocks keeps the matrix rows and the vector
// that neighbours read in shared memory, every other vector in registers,
// gathers across blocks through distributed shared memory, and finishes a
// dot product with one hardware cluster barrier (0.2 us): each block leaves
// its partial sums in its own shared memory, and after the barrier one warp a
// value reads all blocks' partials and adds them in one fixed order, so every
// thread of the cluster holds the same bits and takes the same branches.
// Nothing waits in a spin loop.
//
// Why 256 threads a block, up to eleven cells a thread: the shuffle trees of
// a reduction are bound by the SM's shuffle rate, so a reduction of two
// values takes 0.89 us with 256 threads and 1.25 us with 512 (16 blocks);
// partial sums read after the barrier cost less than remote stores before it
// (a remote load's 0.1 us against 0.3 us for the stores to land).
//
// Measured (us an iteration, the grid kernels' figures in brackets): CG 2.1
// (6.4) at 16^3, 2.3 (6.4) at 16x16x32, 2.9 (6.6) at 24^3, 4.0 (6.7) at 32^3,
// 4.6 (6.8) at 35^3; BiCGStab of three components 5.7 (42) at 16^3, 7.4 at
// 24^3, 9.6 (43) at 32^3.  What bounds it now: the barriers and reductions
// (about 1.3 us of a CG iteration) and, towards 32^3, the gathers (six a cell
// at about 0.3 clocks each a block).
//
// The arithmetic of a cell is that of the grid kernels (CG: the one-reduction
// form of Chronopoulos and Gear as in pcg1_halo_body; BiCGStab: the
// reference's right-preconditioned form with its restarts); only the order of
// the partial sums differs.  BiCGStab components share no data but the
// matrix, so each runs on its own cluster.
#include "gf_krylov.cuh"

#include <mutex>

namespace gf {

constexpr int kClBlocks = 16;   // blocks of the largest cluster (non-portable size)
constexpr int kClThreads = 256;
constexpr int kClValues = 4;    // values of one reduction
constexpr int kClSmemMax = 227 * 1024;

// Dynamic shared memory: the reduction's scratch (every thread's values, the
// block's partials, the totals), then the gathered vector, the coefficients
// and the addresses of the gathered values.
constexpr int kClRedDoubles = kClValues * kClThreads + 2 * 2 * kClValues;
constexpr size_t kClRedBytes = sizeof(double) * kClRedDoubles;
static size_t cl_smem(int64_t chunk, int width) {
    return kClRedBytes + (size_t)chunk * (sizeof(double) + (size_t)width * (sizeof(double) + sizeof(uint32_t)));
}

__device__ __forceinline__ unsigned cl_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cl_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cl_map(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// Ordered against the barriers (volatile), free to overlap with each other.
__device__ __forceinline__ double cl_load(unsigned addr) {
    double v;
    asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void cl_barrier() {
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Cluster-wide sums (max of value 0 with max0) of every thread's NV values:
// the same bits in every thread of the cluster.  Also the barrier between
// what was written before and what is read after.
struct ClReduce {
    double* mine;   // [kClValues][kClThreads] values of this block's threads
    double* part;   // [2][kClValues] this block's partials, read by all blocks
    double* total;  // [2][kClValues]
    unsigned from;  // the partials of block `lane`
    unsigned cs;
    int set;        // used in turn: see below
    __device__ ClReduce(double* s, unsigned size) {
        mine = s;
        part = s + kClValues * kClThreads;
        total = part + 2 * kClValues;
        cs = size;
        const unsigned lane = threadIdx.x & 31;
        from = cl_map((unsigned)__cvta_generic_to_shared(part), lane < size ? lane : 0u);
        set = 0;
    }
    template <int NV>
    __device__ __forceinline__ void run(double (&v)[NV], bool max0) {
        static_assert(NV <= kClValues && NV * 32 <= kClThreads, "one warp a value");
        const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
        for (int j = 0; j < NV; ++j) mine[j * kClThreads + threadIdx.x] = v[j];
        __syncthreads();
        if (warp < NV) {
            const bool mx = warp == 0 && max0;
            double x[kClThreads / 32];
#pragma unroll
            for (int k = 0; k < kClThreads / 32; ++k) x[k] = mine[warp * kClThreads + k * 32 + lane];
#pragma unroll
            for (int h = kClThreads / 64; h > 0; h >>= 1)
#pragma unroll
                for (int k = 0; k < h; ++k) x[k] = comb(x[k], x[k + h], mx);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x[0] = comb(x[0], __shfl_xor_sync(0xffffffffu, x[0], o), mx);
            if (lane == 0) part[set * kClValues + warp] = x[0];
        }
        cl_barrier();
        if (warp < NV) {
            const bool mx = warp == 0 && max0;
            double x = (unsigned)lane < cs ? cl_load(from + 8u * (unsigned)(set * kClValues + warp)) : 0.0;
#pragma unroll
            for (int o = kClBlocks / 2; o > 0; o >>= 1) x = comb(x, __shfl_xor_sync(0xffffffffu, x, o), mx);
            if (lane == 0) total[set * kClValues + warp] = x;
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < NV; ++j) v[j] = total[set * kClValues + j];
        // A block may write the next reduction's partials and totals while a
        // slower one still reads this one's, but not the one after: that lies
        // behind the next barrier.
        set ^= 1;
    }
};

// This block's rows of one system.  Cell i of the block (i = threadIdx.x +
// u * blockDim.x) is cell c0 + i of the system; the neighbour of a slot is
// kept as its address in the cluster's shared memory.
template <int WIDTH, int U>
struct ClRows {
    double* g;  // the gathered vector, own cells
    const double* val;
    const uint32_t* adr;
    int chunk, m, c0;
    int len[U];
    double d[U];

    __device__ void init(const gf_krylov_t& K, char* smem, int chunk_, unsigned rank) {
        chunk = chunk_;
        const int n = (int)K.n;
        c0 = (int)rank * chunk;
        m = n - c0 < chunk ? n - c0 : chunk;
        if (m < 0) m = 0;
        g = reinterpret_cast<double*>(smem + kClRedBytes);
        double* v = g + chunk;
        const int W = WIDTH > 0 ? WIDTH : K.width;
        uint32_t* a = reinterpret_cast<uint32_t*>(v + (size_t)W * chunk);
        val = v;
        adr = a;
        const unsigned gbase = (unsigned)__cvta_generic_to_shared(g);
        const bool box = K.stride_y > 0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = threadIdx.x + u * blockDim.x;
            len[u] = 0;
            d[u] = 0.0;
            if (i >= m) continue;
            const int c = c0 + i;
            d[u] = __ldg(K.diag + c);
            len[u] = WIDTH > 0 ? WIDTH : (K.row_len ? (int)__ldg(K.row_len + c) : K.width);
            for (int s = 0; s < len[u]; ++s) {
                int j;
                double w;
                if (box) {
                    // implicit neighbours; a symmetric matrix has its "-"
                    // coefficients in the "+" slots of the cells below
                    const int st = s < 2 ? 1 : (s < 4 ? (int)K.stride_y : (int)K.stride_z);
                    if (s & 1) {
                        j = c + st < n ? c + st : c;
                        w = __ldg(K.val + (int64_t)s * n + c);
                    } else {
                        j = c >= st ? c - st : c;
                        w = !K.symmetric ? __ldg(K.val + (int64_t)s * n + c)
                                         : (c >= st ? __ldg(K.val + (int64_t)(s + 1) * n + c - st) : 0.0);
                    }
                } else {
                    j = __ldg(K.nbr + (int64_t)s * n + c);
                    w = __ldg(K.val + (int64_t)s * n + c);
                }
                const int rj = j / chunk;
                v[(size_t)s * chunk + i] = w;
                a[(size_t)s * chunk + i] = cl_map(gbase + 8u * (unsigned)(j - rj * chunk), (unsigned)rj);
            }
        }
    }
    __device__ __forceinline__ bool on(int u) const { return (int)(threadIdx.x + u * blockDim.x) < m; }
    __device__ __forceinline__ int local(int u) const { return threadIdx.x + u * blockDim.x; }
    // Row u's product with the gathered vector; gc: its value at the own cell.
    __device__ __forceinline__ double apply(int u, double gc) const {
        const int i = local(u);
        double acc = d[u] * gc;
        if constexpr (WIDTH > 0) {
            double x[WIDTH > 0 ? WIDTH : 1];
#pragma unroll
            for (int s = 0; s < WIDTH; ++s) x[s] = cl_load(adr[s * chunk + i]);
#pragma unroll
            for (int s = 0; s < WIDTH; ++s) acc += val[s * chunk + i] * x[s];
        } else {
            // groups of three slots: a row has six entries as a rule
            for (int s0 = 0; s0 < len[u]; s0 += 3) {
                double x[3];
#pragma unroll
                for (int j = 0; j < 3; ++j) x[j] = s0 + j < len[u] ? cl_load(adr[(s0 + j) * chunk + i]) : 0.0;
#pragma unroll
                for (int j = 0; j < 3; ++j)
                    if (s0 + j < len[u]) acc += val[(s0 + j) * chunk + i] * x[j];
            }
        }
        return acc;
    }
};

__device__ __forceinline__ void cl_stats(double* o, double r0, double fin, int its, int converged, int status) {
    o[0] = r0;
    o[1] = fin;
    o[2] = its;
    o[3] = converged;
    o[4] = status;
}

// Jacobi-PCG with one reduction an iteration: w = A z and the sums |r|, r.z
// and w.z, then the updates of p, q, x, r and z and one barrier that makes z
// visible to the gathers.
template <int WIDTH, int U>
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_cg(const __grid_constant__ gf_krylov_t K, int chunk) {
    extern __shared__ __align__(16) char cl_mem[];
    const unsigned rank = cl_rank(), size = cl_size();
    ClReduce red(reinterpret_cast<double*>(cl_mem), size);
    ClRows<WIDTH, U> rows;
    rows.init(K, cl_mem, chunk, rank);
    const bool jac = K.jacobi != 0, linf = K.norm_inf != 0;
    double x[U], r[U], p[U], q[U], iv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        x[u] = r[u] = p[u] = q[u] = iv[u] = 0.0;
        if (!rows.on(u)) continue;
        x[u] = __ldg(K.x + rows.c0 + rows.local(u));
        iv[u] = inv_diag(K.diag, rows.c0 + rows.local(u), jac);
        rows.g[rows.local(u)] = x[u];
    }
    cl_barrier();
    double loc[2] = {0.0, 0.0};  // this thread's |r| and r.z of the last update
#pragma unroll
    for (int u = 0; u < U; ++u) {
        if (!rows.on(u)) continue;
        r[u] = __ldg(K.rhs + rows.c0 + rows.local(u)) - rows.apply(u, x[u]);
        loc[0] = norm_acc(loc[0], r[u], linf);
        loc[1] += r[u] * (iv[u] * r[u]);
    }
    red.run(loc, linf);  // every gather of x lies before this barrier
    const double r0 = norm_fin(loc[0], linf), thresh = fmax(K.atol, K.rtol * r0);
    double fin = r0, rz = loc[1], alpha = 1.0;
    int its = 0, status = r0 < thresh ? GF_OK : (!isfinite(r0) ? GF_NONFINITE : -1);
    if (K.max_iter <= 0 && status < 0) status = GF_MAX_ITER;
    if (status < 0) {
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (rows.on(u)) rows.g[rows.local(u)] = iv[u] * r[u];
        cl_barrier();
    }
    for (int it = 1; status < 0; ++it) {
        double w[U], sum[3] = {loc[0], loc[1], 0.0};
#pragma unroll
        for (int u = 0; u < U; ++u) {
            w[u] = 0.0;
            if (!rows.on(u)) continue;
            const double z = iv[u] * r[u];
            w[u] = rows.apply(u, z);
            sum[2] += w[u] * z;
        }
        red.run(sum, linf);
        if (it > 1) {
            fin = norm_fin(sum[0], linf);
            its = it - 1;
            if (fin < thresh) status = GF_OK;
            else if (!isfinite(fin)) status = GF_NONFINITE;
            else if (its >= K.max_iter) status = GF_MAX_ITER;
            if (status >= 0) break;
        }
        const double gm = it > 1 ? sum[1] : rz, beta = it > 1 ? gm / rz : 0.0;
        alpha = gm / (it > 1 ? sum[2] - beta * gm / alpha : sum[2]);
        rz = gm;
        loc[0] = loc[1] = 0.0;
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!rows.on(u)) continue;
            p[u] = iv[u] * r[u] + p[u] * beta;
            q[u] = w[u] + q[u] * beta;
            x[u] += alpha * p[u];
            r[u] -= alpha * q[u];
            const double z = iv[u] * r[u];
            rows.g[rows.local(u)] = z;
            loc[0] = norm_acc(loc[0], r[u], linf);
            loc[1] += r[u] * z;
        }
        cl_barrier();
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (rows.on(u)) K.x[rows.c0 + rows.local(u)] = x[u];
    if (rank == 0 && threadIdx.x == 0) cl_stats(K.stats, r0, fin, its, status == GF_OK, status);
    cl_barrier();  // no block leaves while another may read its partials
}

// BiCGStab of one component: five cluster barriers an iteration (v; s; t;
// r; the new direction).  The stopping tests, breakdown tests and restarts
// are those of bicgstab_body, taken by every thread from the same sums.
template <int WIDTH, int U>
__global__ void __launch_bounds__(kClThreads, 1) k_cluster_bicgstab(const __grid_constant__ gf_krylov_t K, int chunk) {
    extern __shared__ __align__(16) char cl_mem[];
    const unsigned rank = cl_rank(), size = cl_size();
    const int comp = (int)(blockIdx.x / size);
    ClReduce red(reinterpret_cast<double*>(cl_mem), size);
    ClRows<WIDTH, U> rows;
    rows.init(K, cl_mem, chunk, rank);
    const bool jac = K.jacobi != 0, linf = K.norm_inf != 0;
    double* gx = K.x + (int64_t)comp * K.n;
    const double* rhs = K.rhs + (int64_t)comp * K.n;
    double x[U], r[U], rh[U], p[U], v[U], s[U], t[U], iv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        x[u] = r[u] = rh[u] = p[u] = v[u] = s[u] = t[u] = iv[u] = 0.0;
        if (!rows.on(u)) continue;
        x[u] = __ldg(gx + rows.c0 + rows.local(u));
        iv[u] = inv_diag(K.diag, rows.c0 + rows.local(u), jac);
        rows.g[rows.local(u)] = x[u];
    }
    cl_barrier();
    BiState st;
    {
        double loc[2] = {0.0, 0.0};
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (!rows.on(u)) continue;
            r[u] = __ldg(rhs + rows.c0 + rows.local(u)) - rows.apply(u, x[u]);
            rh[u] = p[u] = r[u];
            loc[0] = norm_acc(loc[0], r[u], linf);
            loc[1] += r[u] * r[u];
        }
        red.run(loc, linf);
        st.r0 = st.final = norm_fin(loc[0], linf);
        st.thresh = fmax(K.atol, K.rtol * st.r0);
        st.rho_old = loc[1];
        st.restarts = st.its = st.converged = 0;
        st.status = GF_MAX_ITER;
        st.mode = kRun;
        st.alpha = st.omega = st.beta = 0.0;
        if (st.r0 < st.thresh) {
            st.mode = kDone;
            st.converged = 1;
            st.status = GF_OK;
        } else if (!isfinite(st.r0)) {
            st.mode = kDone;
            st.status = GF_NONFINITE;
        }
    }
    // r_hat = p = r after a breakdown; the rest of that iteration is idle.
    auto restart = [&]() {
        double loc[1] = {0.0};
#pragma unroll
        for (int u = 0; u < U; ++u) {
            rh[u] = p[u] = r[u];
            loc[0] += r[u] * r[u];
        }
        red.run(loc, false);
        st.rho_old = loc[0];
        st.mode = kRun;
    };
    for (int it = 1; st.mode == kRun && it <= K.max_iter; ++it) {
        // y = M p, v = A y; r_hat.v, |r_hat|^2, |v|^2
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (rows.on(u)) rows.g[rows.local(u)] = iv[u] * p[u];
        cl_barrier();
        {
            double loc[3] = {0.0, 0.0, 0.0};
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!rows.on(u)) continue;
                v[u] = rows.apply(u, iv[u] * p[u]);
                loc[0] += rh[u] * v[u];
                loc[1] += rh[u] * rh[u];
                loc[2] += v[u] * v[u];
            }
            red.run(loc, false);
            if (fabs(loc[0]) <= 1e-6 * sqrt(loc[1]) * sqrt(loc[2])) breakdown(st, it, K.max_restart);
            else st.alpha = st.rho_old / loc[0];
            if (st.mode == kRestart) {
                restart();
                continue;
            }
            if (st.mode == kDone) break;
        }
        // s = r - alpha v, |s|; z = M s
        {
            double loc[1] = {0.0};
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!rows.on(u)) continue;
                s[u] = r[u] - st.alpha * v[u];
                rows.g[rows.local(u)] = iv[u] * s[u];
                loc[0] = norm_acc(loc[0], s[u], linf);
            }
            red.run(loc, linf);
            const double fin = norm_fin(loc[0], linf);
            st.final = fin;
            if (fin < st.thresh) {
#pragma unroll
                for (int u = 0; u < U; ++u) x[u] += st.alpha * (iv[u] * p[u]);
                st.mode = kDone;
                st.converged = 1;
                st.its = it;
                st.status = GF_OK;
                break;
            }
            if (!isfinite(fin)) {
                st.mode = kDone;
                st.its = it;
                st.status = GF_NONFINITE;
                break;
            }
        }
        // t = A z; t.t, t.s
        {
            double loc[2] = {0.0, 0.0};
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!rows.on(u)) continue;
                t[u] = rows.apply(u, iv[u] * s[u]);
                loc[0] += t[u] * t[u];
                loc[1] += t[u] * s[u];
            }
            red.run(loc, false);
            const double dd = loc[0], tn = sqrt(loc[0]);
            if (fabs(dd) <= 1e-6 * tn * tn) {
                breakdown(st, it, K.max_restart);
            } else {
                st.omega = loc[1] / dd;
                if (fabs(st.omega) <= 1e-6) breakdown(st, it, K.max_restart);
            }
            if (st.mode == kRestart) {
                restart();
                continue;
            }
            if (st.mode == kDone) break;
        }
        // x += alpha y + omega z, r = s - omega t; |r|, r_hat.r, |r_hat|^2, |r|^2
        {
            double loc[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!rows.on(u)) continue;
                x[u] = x[u] + st.alpha * (iv[u] * p[u]) + st.omega * (iv[u] * s[u]);
                r[u] = s[u] - st.omega * t[u];
                loc[0] = norm_acc(loc[0], r[u], linf);
                loc[1] += rh[u] * r[u];
                loc[2] += rh[u] * rh[u];
                loc[3] += r[u] * r[u];
            }
            red.run(loc, linf);
            const double fin = norm_fin(loc[0], linf);
            st.final = fin;
            if (fin < st.thresh) {
                st.mode = kDone;
                st.converged = 1;
                st.its = it;
                st.status = GF_OK;
                break;
            }
            if (!isfinite(fin)) {
                st.mode = kDone;
                st.its = it;
                st.status = GF_NONFINITE;
                break;
            }
            if (fabs(loc[1]) <= 1e-6 * sqrt(loc[2]) * sqrt(loc[3])) {
                breakdown(st, it, K.max_restart);
                if (st.mode == kDone) break;
                restart();
                continue;
            }
            st.beta = (loc[1] / st.rho_old) * (st.alpha / st.omega);
            st.rho_old = loc[1];
        }
        // p = r + beta (p - omega v)
#pragma unroll
        for (int u = 0; u < U; ++u) p[u] = r[u] + st.beta * (p[u] - st.omega * v[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
        if (rows.on(u)) gx[rows.c0 + rows.local(u)] = x[u];
    if (rank == 0 && threadIdx.x == 0) {
        const bool fin = st.mode == kDone;
        cl_stats(K.stats + 5 * comp, st.r0, st.final, fin ? st.its : K.max_iter, st.converged,
                 fin ? st.status : GF_MAX_ITER);
    }
    cl_barrier();  // no block leaves while another may read its partials
}

// ---------------------------------------------------------------------------
// Cells a thread can hold: the CG keeps seven doubles a cell in registers and
// BiCGStab nine, of the 255 registers a thread has at 256 threads a block.
constexpr int kClMaxU[2] = {11, 8};

// Whether a cluster of kClBlocks blocks with the largest shared memory can
// run on the current device (a partitioned GPU may not have one), asked once
// a device.
static bool cluster_available() {
    static std::mutex mu;
    static signed char known[128] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) return false;
    std::lock_guard<std::mutex> lock(mu);
    if (known[dev] == 0) {
        const void* kern = (const void*)k_cluster_cg<6, 11>;
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = kClBlocks;
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(kClBlocks);
        cfg.blockDim = dim3(kClThreads);
        cfg.dynamicSmemBytes = kClSmemMax;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        int n = 0;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kClSmemMax);
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
        known[dev] = e == cudaSuccess && n >= 1 ? 1 : -1;
        if (e != cudaSuccess) (void)cudaGetLastError();  // not an error of the caller's solve
    }
    return known[dev] > 0;
}

bool cluster_fits(const gf_krylov_t& k, bool bicgstab) {
    // A caller that bounds the blocks or the waits asks for the kernels that
    // honour those bounds (a cluster barrier has no poll limit).
    if (k.mixed || k.single_reduction || k.block_cap > 0 || k.spin_limit > 0) return false;
    if (!bicgstab && k.ncomp != 1) return false;
    // The largest system: its rows (80 bytes a cell at width 6) in 16 blocks'
    // shared memory and its vectors in their registers, up to 44,816 cells for
    // the CG (2,801 a block) and 32,768 for BiCGStab.  There the cluster is still the faster
    // (CG 4.6 against 6.8 us at 42,875 cells, BiCGStab 9.6 against 43).
    const int64_t chunk = (k.n + kClBlocks - 1) / kClBlocks;
    return chunk <= (int64_t)kClMaxU[bicgstab] * kClThreads && cl_smem(chunk, k.width) <= (size_t)kClSmemMax &&
           cluster_available();
}

template <int WIDTH>
static const void* cl_kernel(int u, bool bicgstab) {
    if (bicgstab)
        return u <= 1 ? (const void*)k_cluster_bicgstab<WIDTH, 1>
                      : (u <= 2 ? (const void*)k_cluster_bicgstab<WIDTH, 2>
                                : (u <= 4 ? (const void*)k_cluster_bicgstab<WIDTH, 4>
                                          : (const void*)k_cluster_bicgstab<WIDTH, 8>));
    return u <= 1 ? (const void*)k_cluster_cg<WIDTH, 1>
                  : (u <= 2 ? (const void*)k_cluster_cg<WIDTH, 2>
                            : (u <= 4 ? (const void*)k_cluster_cg<WIDTH, 4>
                                      : (u <= 8 ? (const void*)k_cluster_cg<WIDTH, 8>
                                                : (const void*)k_cluster_cg<WIDTH, 11>)));
}

int launch_cluster(const gf_krylov_t* k, bool bicgstab, cudaStream_t st) {
    // One cell a thread as long as there are blocks: a cluster of one block
    // up to 256 cells, then twice the blocks for twice the cells up to 16.
    int size = 1;
    while (size < kClBlocks && (int64_t)size * kClThreads < k->n) size *= 2;
    int chunk = (int)((k->n + size - 1) / size);
    const int u = (chunk + kClThreads - 1) / kClThreads;
    const void* kern = k->width == 6 ? cl_kernel<6>(u, bicgstab) : cl_kernel<0>(u, bicgstab);
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)size;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(size * (bicgstab ? k->ncomp : 1)));
    cfg.blockDim = dim3((unsigned)kClThreads);
    cfg.dynamicSmemBytes = cl_smem(chunk, k->width);
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    gf_krylov_t arg = *k;
    void* args[] = {&arg, &chunk};
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kClSmemMax);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e == cudaSuccess) e = cudaLaunchKernelExC(&cfg, kern, args);
    if (e != cudaSuccess) {
        set_error("%s: cluster launch failed: %s", bicgstab ? "gf_bicgstab_solve" : "gf_pcg_solve",
                  cudaGetErrorString(e));
        return GF_ERR_CUDA;
    }
    return GF_OK;
}

}  // namespace gf
