// Barrier and reduction of a persistent cooperative launch (or of one system's
// share of its blocks), for kernels whose blocks hold at most one block an SM.
#pragma once

#include "gf_krylov.cuh"

namespace gf {

template <int T, int NVMAX>
struct GridShared {
    static constexpr int kThreads = T;
    static constexpr int kSlots = T > 512 ? T / 2 : T;  // per value in shared memory
    // barrier state of this block's system
    unsigned epoch;
    int nblk, bid, err;
    long long spin;
    // a reduction's totals and the threads' values
    double total[NVMAX];
    double mine[NVMAX * kSlots];
};

// Arrive and wait for all blocks of the system (bounded; false: gave up, or
// another block did).  The CTA barriers make the release cumulative over the
// block's writes and order its later reads behind the acquire.
template <int T, int NVMAX>
__device__ __forceinline__ bool grid_sync(GridShared<T, NVMAX>& sh, KCtl* ctl) {
    __syncthreads();
    if (threadIdx.x < 32) {
        const unsigned ep = sh.epoch;
        __syncwarp();
        if (threadIdx.x == 0) arrive_release(&ctl->count);
        const unsigned long long target = (unsigned long long)(ep + 1u) * (unsigned)sh.nblk;
        int err = 0;
        long long it = 0;
        while (true) {
            const unsigned long long c = load_acquire(&ctl->count);
            if (__all_sync(0xffffffffu, c >= target)) break;
            __nanosleep(20);
            ++it;
            if ((it & 255) == 0 && __any_sync(0xffffffffu, vload(&ctl->error) != 0)) {
                err = 1;
                break;
            }
            if (it > sh.spin) {
                if (threadIdx.x == 0) atomicExch(&ctl->error, 1);
                err = 1;
                break;
            }
        }
        if (threadIdx.x == 0) {
            sh.err = err;
            sh.epoch = ep + 1u;
        }
    }
    __syncthreads();
    return sh.err == 0;
}

// Sums over all blocks of NV values a thread (max where maxmask has the bit
// set), and the barrier.  The totals are left in total (what was there before
// stays when the wait gave up); every block adds the blocks' partials in the
// same fixed order.
template <int NV, int T, int NVMAX>
__device__ __forceinline__ bool grid_sum(GridShared<T, NVMAX>& sh, KCtl* ctl, double* partials, double (&v)[NV], unsigned maxmask) {
    constexpr int kSlots = GridShared<T, NVMAX>::kSlots, kPer = kSlots / 32, kLoads = 5;
    static_assert(NV <= NVMAX && 32 * NV <= T, "one warp a value");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // double-buffered by barrier parity (see kPartials)
    double* part = partials + (sh.epoch & 1u) * (kPartials / 2);
#pragma unroll
    for (int j = 0; j < NV; ++j) {
        if constexpr (T > 512) {
            v[j] = comb(v[j], __shfl_xor_sync(0xffffffffu, v[j], 16), (maxmask >> j) & 1u);
            if (lane < 16) sh.mine[j * kSlots + warp * 16 + lane] = v[j];
        } else {
            sh.mine[j * kSlots + threadIdx.x] = v[j];
        }
    }
    __syncthreads();
    const bool mx = (maxmask >> warp) & 1u;
    if (warp < NV) {
        double x[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) x[k] = sh.mine[warp * kSlots + k * 32 + lane];
#pragma unroll
        for (int h = kPer / 2; h > 0; h >>= 1)
#pragma unroll
            for (int k = 0; k < h; ++k) x[k] = comb(x[k], x[k + h], mx);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x[0] = comb(x[0], __shfl_xor_sync(0xffffffffu, x[0], o), mx);
        if (lane == 0) __stcg(part + (int64_t)warp * kMaxBlocks + sh.bid, x[0]);
    }
    if (!grid_sync(sh, ctl)) return false;
    if (warp < NV) {
        // Every load of a lane issued before any is added: in a plain loop the
        // five L2 round trips follow one another (3.4 us a reduction of 148
        // blocks against 2.1).
        const int nblk = sh.nblk;
        double x = 0.0;  // the identity of both: the max values are norms
        for (int b0 = lane; b0 < nblk; b0 += 32 * kLoads) {
            double y[kLoads];
#pragma unroll
            for (int q = 0; q < kLoads; ++q) {
                const int b = b0 + 32 * q;
                y[q] = b < nblk ? __ldcg(part + (int64_t)warp * kMaxBlocks + b) : 0.0;
            }
#pragma unroll
            for (int q = 0; q < kLoads; ++q) x = comb(x, y[q], mx);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x = comb(x, __shfl_xor_sync(0xffffffffu, x, o), mx);
        if (lane == 0) sh.total[warp] = x;
    }
    __syncthreads();
    return true;
}

// Sets the barrier state of block bid of nblk; a CTA barrier must follow.
template <int T, int NVMAX>
__device__ __forceinline__ void grid_init(GridShared<T, NVMAX>& sh, const gf_krylov_t& K, int nblk, int bid) {
    if (threadIdx.x == 0) {
        sh.epoch = 0;
        sh.nblk = nblk;
        sh.bid = bid;
        sh.err = 0;
        sh.spin = K.spin_limit > 0 ? K.spin_limit : kSpinLimit;
    }
}

}  // namespace gf
