// Shared device helpers for the cat-surface B200 kernels.
//
// Everything here is plain CUDA C++ for sm_100a: cache-hinted loads/stores,
// a bounded grid barrier for persistent cooperative kernels, and the status
// word every persistent kernel reports through.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "../../include/catsurf_b200.h"

namespace csg {

// Correctly rounded x / 3 for finite binary64 x with |x| >= 2^-1000 (far from
// the subnormal range, where RN(x zl) loses the needed bits) with two
// multiplies (Brisebarre, Muller and Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", IEEE TC
// 53(8), 2004): q = RN(x zh + RN(x zl)) with zh = RN(1/3) and
// zl = RN(1/3 - zh) = zh * 2^-54.  Why it is exact for the divisor 3: the
// exact quotient x/3 = M 2^e / 3 sits at a multiple of a third of a unit in
// the last place, so it is never closer than 1/6 ulp to a rounding midpoint,
// while x zh + RN(x zl) is within ~2^-105 relative of x/3.  Equal to
// __ddiv_rn(x, 3.0) bit for bit (csg_selftest_div3 and the sweep and
// preprocess tests, which compare against the oracle's plain division).
__device__ __forceinline__ double div3_rn(double x) {
    const double zh = 0x1.5555555555555p-2;
    const double zl = 0x1.5555555555555p-56;
    return __fma_rn(x, zh, __dmul_rn(x, zl));
}

// Status word layout inside a kernel's control block (first 256 bytes of its
// scratch).  word 0: barrier arrival counter; word 1: status (CSG_OK or a
// negative CSG_ERR_*); word 2: index of the barrier/step that failed.
struct Control {
    unsigned int arrivals;
    int status;
    int where;
    int pad[61];
};
static_assert(sizeof(Control) == 256, "control block is 256 bytes");

__device__ __forceinline__ unsigned long long global_timer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned int ld_acquire_gpu(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ int ld_relaxed_gpu(const int* p) {
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void red_release_gpu_add(unsigned int* p, unsigned int v) {
    asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Grid-wide barrier for a cooperatively launched (all CTAs co-resident)
// kernel.  `phase` counts the arrivals expected so far and must be advanced
// identically by every CTA.  Waits are bounded by `timeout_ns`; on timeout or
// when another CTA has already reported an error the barrier returns true
// and the caller must leave the kernel.  No trap, no unbounded spin.
// Ordering: __syncthreads orders the CTA's writes before thread 0's arrival,
// a release at gpu scope (cumulative, so it covers what thread 0 has
// observed through the CTA barrier); the acquire poll and the closing
// __syncthreads order the other CTAs' writes before this CTA's next reads.
__device__ __forceinline__ bool grid_barrier(Control* ctl, unsigned int& phase, unsigned long long timeout_ns,
                                             int where) {
    __shared__ int s_abort;
    __syncthreads();
    phase += gridDim.x;
    if (threadIdx.x == 0) {
        red_release_gpu_add(&ctl->arrivals, 1u);
        int abort = 0;
        unsigned long long start = global_timer_ns();
        unsigned int polls = 0;
        while (true) {
            unsigned int seen = ld_acquire_gpu(&ctl->arrivals);
            if (static_cast<int>(seen - phase) >= 0) break;
            if (((++polls) & 31u) == 0u) {
                if (ld_relaxed_gpu(&ctl->status) != CSG_OK) { abort = 1; break; }
                if (global_timer_ns() - start > timeout_ns) {
                    if (atomicCAS(&ctl->status, CSG_OK, CSG_ERR_TIMEOUT) == CSG_OK) ctl->where = where;
                    abort = 1;
                    break;
                }
            }
        }
        s_abort = abort;
    }
    __syncthreads();
    return s_abort != 0;
}

// Published words of the dataflow kernels: 16 bytes that hold a value (three
// float32 coordinates, or a float64) and the number of updates it belongs to.  A
// .b128 access with .relaxed is one scalar memory operation (PTX ISA 8.3, sm_70
// and later), so a load returns a value together with its own version and needs
// no acquire ordering.
struct alignas(16) Quad {
    unsigned long long lo, hi;
};
__device__ __forceinline__ Quad ld_quad(const Quad* p) {
    Quad q;
    asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
                 : "=l"(q.lo), "=l"(q.hi)
                 : "l"(p)
                 : "memory");
    return q;
}
__device__ __forceinline__ void st_quad(Quad* p, const Quad& q) {
    asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}" ::"l"(p),
                 "l"(q.lo), "l"(q.hi)
                 : "memory");
}
__device__ __forceinline__ Quad make_quad(float x, float y, float z, unsigned int version) {
    return {(static_cast<unsigned long long>(__float_as_uint(y)) << 32) | __float_as_uint(x),
            (static_cast<unsigned long long>(version) << 32) | __float_as_uint(z)};
}
__device__ __forceinline__ unsigned int quad_version(const Quad& q) { return static_cast<unsigned>(q.hi >> 32); }
__device__ __forceinline__ float4 quad_point(const Quad& q) {
    return make_float4(__uint_as_float(static_cast<unsigned>(q.lo)), __uint_as_float(static_cast<unsigned>(q.lo >> 32)),
                       __uint_as_float(static_cast<unsigned>(q.hi)), 0.0f);
}

// x[0] + x[1] + ... + x[n - 1] in that order, starting from 0 (the blocked sums fold their
// partials so, whatever the launch shape), by one CTA of kOrderedThreads; the sum is valid
// in thread 0.  `buf` holds kOrderedChunk elements.  One thread reading global memory pays
// a round trip every few elements (960 partials: 37 us); here the CTA brings a chunk into
// shared memory at once and the chain of additions runs from there (960: 8 us).
constexpr int kOrderedThreads = 256, kOrderedChunk = 1024;
template <typename T>
__device__ __forceinline__ T ordered_sum(const T* __restrict__ x, int n, T* buf) {
    T sum = T(0);
    for (int base = 0; base < n; base += kOrderedChunk) {
        const int m = min(kOrderedChunk, n - base);
        __syncthreads();
        for (int i = threadIdx.x; i < m; i += blockDim.x) buf[i] = x[base + i];
        __syncthreads();
        if (threadIdx.x == 0) {
            int i = 0;
            for (; i + 8 <= m; i += 8)
#pragma unroll
                for (int k = 0; k < 8; ++k) sum = sum + buf[i + k];
            for (; i < m; ++i) sum = sum + buf[i];
        }
    }
    return sum;
}

// Bounded wait of one warp in a dataflow kernel: every 64 polls (`polls` is the
// same in every lane) lane 0 checks the clock and the status word; true (the
// same in every lane) means give up -- the status is CSG_ERR_TIMEOUT (recorded
// here) or another CTA's error.
__device__ __forceinline__ bool warp_wait_expired(Control* ctl, unsigned long long timeout_ns, unsigned int& polls,
                                                  unsigned long long& start) {
    if (((++polls) & 63u) != 0u) return false;
    int expired = 0;
    if ((threadIdx.x & 31) == 0) {
        const unsigned long long now = global_timer_ns();
        if (start == 0) start = now;
        if (ld_relaxed_gpu(&ctl->status) != CSG_OK) {
            expired = 1;
        } else if (now - start > timeout_ns) {
            if (atomicCAS(&ctl->status, CSG_OK, CSG_ERR_TIMEOUT) == CSG_OK) ctl->where = -2;
            expired = 1;
        }
    }
    return __shfl_sync(0xffffffffu, expired, 0) != 0;
}

}  // namespace csg
