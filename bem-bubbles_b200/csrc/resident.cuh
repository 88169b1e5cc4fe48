// Pieces of the kernels whose vectors stay on the SMs (bicg_resident.cu, refine_resident.cu): one CTA of RB_T
// threads per SM, every CTA holds all of each vector, thread t its elements t + k RB_T.
#pragma once

#include "slots.cuh"

namespace bemb {

constexpr int RB_T = 512;
constexpr int RB_WARPS = RB_T / 32;
constexpr int RB_SMEM = 226 * 1024;  // dynamic shared memory of a CTA, at most

// Two sums over the CTA's threads, the same bits in every thread and, from the same inputs, in
// every CTA; false when some thread's exchange wait expired (!ok).  rs: 2 RB_WARPS doubles, written again only
// after another barrier of the CTA.
__device__ __forceinline__ bool cta_sums(double* rs, double u, double w, bool ok, double& su, double& sw) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        u += __shfl_xor_sync(0xffffffffu, u, o);
        w += __shfl_xor_sync(0xffffffffu, w, o);
    }
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) {
        rs[wid] = u;
        rs[RB_WARPS + wid] = w;
    }
    const bool bad = __syncthreads_or(!ok);
    u = rs[lane & (RB_WARPS - 1)];
    w = rs[RB_WARPS + (lane & (RB_WARPS - 1))];
#pragma unroll
    for (int o = RB_WARPS / 2; o > 0; o >>= 1) {
        u += __shfl_xor_sync(0xffffffffu, u, o);
        w += __shfl_xor_sync(0xffffffffu, w, o);
    }
    su = u;
    sw = w;
    return !bad;
}

// The thread's elements (tid + k RB_T) of the vector published in `slots` under seq; false (the whole warp)
// when a wait ran out.  The warp polls as
// one: lanes that leave the loop apart would run what follows in as many passes.
template <int K>
__device__ __forceinline__ bool collect(const ulonglong2* slots, int n, unsigned long long seq, long long limit,
                                        double (&v)[K]) {
    constexpr int B = K < 4 ? K : 4;  // loads in flight
    const long long t0 = clock64();
#pragma unroll
    for (int k0 = 0; k0 < K; k0 += B) {
        unsigned pend = 0;
#pragma unroll
        for (int k = 0; k < B; ++k) {
            v[k0 + k] = 0.0;
            if ((int)threadIdx.x + (k0 + k) * RB_T < n) pend |= 1u << k;
        }
        while (__any_sync(0xffffffffu, pend)) {
            unsigned long long lo[B], hi[B];
#pragma unroll
            for (int k = 0; k < B; ++k)
                if (pend >> k & 1) slot_load(slots + threadIdx.x + (k0 + k) * RB_T, lo[k], hi[k]);
#pragma unroll
            for (int k = 0; k < B; ++k)
                if ((pend >> k & 1) && hi[k] == seq) {
                    v[k0 + k] = __longlong_as_double((long long)lo[k]);
                    pend &= ~(1u << k);
                }
            if (__any_sync(0xffffffffu, pend && clock64() - t0 > limit)) return false;
        }
    }
    return true;
}

// 16 bytes (two rows of a column) into the thread's own ring slot, through L2 only; `in` false: zeros.
__device__ __forceinline__ void ring_copy(double2* slot, const double* src, bool in, uint64_t pol) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2, %3;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(slot)),
                 "l"(src), "r"(in ? 16 : 0), "l"(pol)
                 : "memory");
}

}  // namespace bemb
