// mailbox.cuh -- the messages that blocks of the resident kernel exchange
// through global memory (step_resident.cuh), and the bounded wait for them.
#pragma once

#include "resident_launch.h"

namespace fomo {

// One 16-byte message; each half is written and read as one 64-bit access.
__device__ __forceinline__ void mail_put(ulonglong2* p, float a, float b, uint32_t tag) {
    const uint64_t lo = ((uint64_t)tag << 32) | __float_as_uint(a), hi = ((uint64_t)tag << 32) | __float_as_uint(b);
    asm volatile("st.relaxed.gpu.global.v2.b64 [%0], {%1, %2};" ::"l"(p), "l"(lo), "l"(hi) : "memory");
}
__device__ __forceinline__ ulonglong2 mail_get(const ulonglong2* p) {
    ulonglong2 v;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
    return v;
}
constexpr int kMailPolls = 1 << 22;

// Whether a wait for messages gives up at poll number `it` (asked at every
// 4096th poll): past `limit` polls, or when another block has given up.  The
// status word then says so.
__device__ __forceinline__ bool mail_check_due(int it) { return (it & 4095) == 4095; }
__device__ __forceinline__ bool mail_gives_up(int it, int limit, int* status) {
    if (it >= limit || *reinterpret_cast<volatile int*>(status) != 0) {
        atomicCAS(status, 0, kErrResidentTimeout);
        return true;
    }
    return false;
}

// Self-test of that wait: one thread polls a message that nobody sends.
static __global__ void mail_selftest_kernel(const ulonglong2* box, int* status, int limit) {
    if (threadIdx.x != 0) return;
    for (int it = 0; (uint32_t)(mail_get(box).x >> 32) != 1u; ++it)
        if (mail_check_due(it) && mail_gives_up(it, limit, status)) return;
}

}  // namespace fomo
