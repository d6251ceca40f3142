// cgsum.cuh -- sums over a thread-block cluster for the conjugate-gradient
// kernels (coulomb.cu, mixing.cu).
//
// Their iterations are chains of latencies (an FP64 add takes 64 clocks, a
// divide 549, a cluster barrier 400), so a sum takes few dependent adds, two
// sums share one chain, and the cluster meets once.
#pragma once

#include <stdint.h>

namespace mg {

constexpr int kCluster = 8;   // blocks of a cluster of the CG kernels

// Sums of x and of y over the warp in one chain of five adds: after the first
// exchange the lower half-warp carries x, the upper one y.  Lane 0 ends with
// the sum of x, lane 16 with that of y.
__device__ __forceinline__ double warp_sum2(double x, double y) {
    const bool up = (threadIdx.x & 16) != 0;
    double v = (up ? y : x) + __shfl_xor_sync(0xffffffffu, up ? x : y, 16);
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// 1 / d by Newton's iteration from the float reciprocal (a CG coefficient:
// right to an ulp or two; an FP64 divide takes 549 clocks).  The float comes
// and goes by bit moves, as FP64 conversions wait for the FP64 pipe.
__device__ __forceinline__ double inverse(double d) {
    const unsigned hi = (unsigned)__double2hiint(d), e = (hi >> 20) & 0x7FFu;
    if (e < 1023 - 100 || e > 1023 + 100) return 1.0 / d;
    float f = __uint_as_float((hi & 0x80000000u) | ((hi & 0x7FFFFFFFu) - (896u << 20)) << 3 |
                              (unsigned)__double2loint(d) >> 29);
    asm("rcp.approx.ftz.f32 %0, %0;" : "+f"(f));
    const unsigned u = __float_as_uint(f);
    double x = __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7FFFFFFFu) >> 3) + (896u << 20))),
                                (int)(u << 29));
    x = fma(x, fma(-d, x, 1.0), x);
    return fma(x, fma(-d, x, 1.0), x);
}

// What the blocks of a cluster leave in each other's shared memory.
struct ClusterSum {
    double part[2][2][kCluster];   // [turn][x, y][rank]: the ranks' partial sums
    int bad[2][kCluster];          // `fail` of that rank
    double warp[2][16];
    double result[2];
    int fail;                      // this block gives up
    int late;                      // sums of other clusters did not come to this block
};

// The address of the same shared variable in the block `rank` of the cluster.
__device__ __forceinline__ uint32_t remote(const void* p, int rank) {
    uint32_t a = (uint32_t)__cvta_generic_to_shared(p), r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void put_remote(uint32_t a, double x) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(x) : "memory");
}

// Whether the kernel runs in clusters of kCluster blocks, as its attribute
// asks: without them there is no other rank to write to.
__device__ __forceinline__ bool in_cluster() {
    uint32_t n;
    asm("mov.u32 %0, %%cluster_nctaid.x;" : "=r"(n));
    return n == (uint32_t)kCluster;
}

__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Sums x and y over the cluster (blocks of at most 512 threads): warp 0 of
// every rank gets the totals in x and y.  `meanwhile` is work of warp 0 for the
// time that the barrier takes.  False, on all ranks alike, when one of them has
// set its `fail`; threads that have left count as arrived at the barrier.
template <class Meanwhile>
__device__ bool cluster_sum(ClusterSum& S, int turn, int rank, double& x, double& y,
                            Meanwhile meanwhile) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    double v = warp_sum2(x, y);
    if (nw > 1) {
        if ((lane & 15) == 0) S.warp[lane >> 4][warp] = v;
        __syncthreads();
        if (warp == 0) {
            v = (lane & 15) < nw ? S.warp[lane >> 4][lane & 15] : 0.0;
#pragma unroll
            for (int o = 8; o > 0; o >>= 1)
                if (o < nw) v += __shfl_xor_sync(0xffffffffu, v, o);
        }
    } else {
        __syncwarp();   // `fail` of any lane
    }
    if (warp == 0) {
        // lane r of the lower half sends x, of the upper half y, to rank r
        v = __shfl_sync(0xffffffffu, v, lane & 16);
        if ((lane & 15) < kCluster) {
            put_remote(remote(&S.part[turn][lane >> 4][rank], lane & 15), v);
            if (lane < kCluster)
                asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(remote(&S.bad[turn][rank], lane)),
                             "r"(S.fail)
                             : "memory");
        }
    }
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    if (warp == 0) meanwhile();
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    int bad = 0;
#pragma unroll
    for (int r = 0; r < kCluster; ++r) bad |= S.bad[turn][r];
    if (bad) return false;
    if (warp == 0) {
        v = S.part[turn][lane >> 4][lane % kCluster];
#pragma unroll
        for (int o = kCluster / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        x = __shfl_sync(0xffffffffu, v, 0);
        y = __shfl_sync(0xffffffffu, v, 16);
    }
    return true;
}

}  // namespace mg
