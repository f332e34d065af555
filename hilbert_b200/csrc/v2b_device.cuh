// Device building blocks for the B200 v2RDM path (sm_100a).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace v2b {

constexpr uint32_t kDevColMask = (1u << 27) - 1u;
constexpr int kStatusTimeout = 4;   // V2B_DEVICE_TIMEOUT
constexpr int kStatusNan = 3;       // V2B_NAN

// the GPU's nanosecond clock (PTX %globaltimer)
__device__ __forceinline__ unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Deterministic block reduction (fixed tree); result valid in thread 0.
__device__ __forceinline__ double block_sum(double v, double *red /* >= 32 */) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double s = 0.0;
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        s = lane < nw ? red[lane] : 0.0;
        s = warp_sum(s);
    }
    return s;
}

__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_down_sync(0xffffffffu, v, o));
    return v;
}

// Block max; result valid in thread 0.
__device__ __forceinline__ double block_max(double v, double *red /* >= 32 */) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    v = warp_max(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double s = 0.0;
    if (wid == 0) {
        const int nw = (blockDim.x + 31) >> 5;
        s = lane < nw ? red[lane] : 0.0;
        s = warp_max(s);
    }
    return s;
}

__device__ __forceinline__ int ld_volatile_i32(const int *p) { return *((volatile const int *)p); }
__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int *p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ unsigned int atom_add_release_u32(unsigned int *p, unsigned int v) {
    unsigned int old;
    asm volatile("atom.add.release.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// Grid-wide barrier of a cooperatively launched kernel that also sums partial
// values over the grid.  A CTA stores its partials in their slots, counts
// itself in with release and polls the count, which only grows (no reset, no
// generation word), then reads every slot; two sets of slots take turns,
// because a CTA past a barrier fills its next slots while others still read.
// The sum runs over the slots in a fixed order: the same bits on every CTA and
// in every run.  2.2 us over 148 CTAs, 1.7 us over 15 (one thread of each
// polls one word; slots polled as the arrival flags themselves took 5.1 us
// and 1.7 us).  Waits are bounded: after spin_limit polls the CTA records
// kStatusTimeout in *status, and every CTA leaves at its next barrier.
struct GridSum {
    double *slots;               // 2 x nslots
    int nslots;
    unsigned int *count;         // 0 at launch
    int *status;
    long long spin_limit;
    double *total;               // shared, 1
    int *fail;                   // shared, 0 at first use
    unsigned int seq;            // barriers passed

    __device__ __forceinline__ double *set() const { return slots + (seq & 1u) * (size_t)nslots; }
    // Called by warp 0 after the CTA's partials were stored in set() (by this
    // warp) and __syncthreads() has ordered the CTA's other writes before it.
    __device__ __forceinline__ void arrive_and_sum(int lane) {
        const double *part = set();
        if (gridDim.x > 1 && lane == 0) {
            atom_add_release_u32(count, 1u);
            const unsigned int want = (seq + 1u) * gridDim.x;
            long long spins = 0;
            while ((int)(ld_acquire_u32(count) - want) < 0) {
                if ((spins & 63) == 0 && ld_volatile_i32(status) != 0) { *fail = 1; break; }
                if (++spins > spin_limit) {
                    atomicExch(status, kStatusTimeout);
                    *fail = 1;
                    break;
                }
                if (spins > 256) __nanosleep(32);
            }
        }
        __syncwarp();
        double s = 0.0;
#pragma unroll 4
        for (int i = lane; i < nslots; i += 32) s += __ldcg(part + i);
        s = warp_sum(s);
        if (lane == 0) *total = s;
    }
    // every thread, after a __syncthreads(): false when the kernel must stop
    // (timeout or an error status)
    __device__ __forceinline__ bool done(double &sum) {
        seq++;
        sum = *total;
        return *fail == 0;
    }
};

// Round-robin ("circle method") pairing of np (even) indices: in step s the
// fixed index np-1 meets s and, for k >= 1, (s+k) meets (s-k) mod (np-1).
__device__ __forceinline__ void rr_pair(int s, int k, int np, int &p, int &q) {
    const int m1 = np - 1;
    int a, b;
    if (k == 0) {
        a = m1;
        b = s;
    } else {
        a = (s + k) % m1;
        b = (s - k + m1) % m1;
    }
    p = a < b ? a : b;
    q = a < b ? b : a;
}

}  // namespace v2b
