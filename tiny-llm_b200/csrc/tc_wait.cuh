// A barrier wait that gives up: what a lost arrival leads to in the TMA-fed kernels.
//
// A wait past its limit marks the CTA (a flag in its shared memory, which ends all its further waits at once), and the kernel's count,
// which the host can read, goes up.  The roles of a marked CTA issue nothing more and store NaN for every row they have not finished, and
// the CTA frees its tensor memory after its copies in flight have had time to land.  So the event never ends in a hung GPU, a lost context or
// numbers that look right.
#pragma once

#include "tc05.cuh"

namespace tl {

static __device__ unsigned int g_gave_up;  // of this translation unit's kernels

// -1: cannot be read.  Another thread may be capturing a graph, which a copy in the default mode would break.
static inline long long read_gave_up() {
    unsigned int n = 0;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    if (cudaThreadExchangeStreamCaptureMode(&mode) != cudaSuccess) return -1;
    const bool ok = cudaMemcpyFromSymbol(&n, g_gave_up, sizeof(n)) == cudaSuccess;
    if (!ok) cudaGetLastError();
    cudaThreadExchangeStreamCaptureMode(&mode);
    return ok ? static_cast<long long>(n) : -1;
}

// Whole warps; the answer is the same in all lanes: whether the phase is over.  false: the CTA is marked.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity, volatile int *dead, uint32_t limit = 1u << 22) {
    for (uint32_t spins = 0;; ++spins) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (__all_sync(0xffffffffu, done)) return true;
        if (__any_sync(0xffffffffu, *dead)) return false;
        if (spins > limit) {
            if ((threadIdx.x & 31) == 0) {
                *dead = 1;
                atomicAdd(&g_gave_up, 1u);
            }
            __syncwarp();
            return false;
        }
    }
}

// The factor on a row's numbers when they are stored, read after the last wait they depend on.
__device__ __forceinline__ float tc_verdict(bool ok, const volatile int *dead) { return ok && !*dead ? 1.f : __int_as_float(0x7fffffff); }

// The last thing before a CTA frees its tensor memory, with all its warps past their loops.
__device__ __forceinline__ void tc_settle(const volatile int *dead) {
    if (*dead)
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
}

}  // namespace tl
