// Loads of memory that others may still be writing when the kernel starts.
//
// A kernel launched ahead of its turn (programmatic dependent launch) is on the
// GPU while the grid before it still writes, and waits for it inside
// (griddepcontrol.wait).  What that grid writes is then not read-only for the
// kernel's lifetime, which is what __ldg and const __restrict__ promise: such a
// load may be taken from ahead of the wait.  Behind the wait these words are read
// by ld_prior, an ordinary load at this point of the program; so are the flags and
// counts that other CTAs of the same launch write, by ld_l2, past L1.
#pragma once

#include <cstdint>

namespace wk {
namespace dev {

__device__ __forceinline__ int32_t ld_prior(const int32_t *p) {
    int32_t v;
    asm volatile("ld.global.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld_prior(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int64_t ld_prior(const int64_t *p) {
    int64_t v;
    asm volatile("ld.global.s64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned long long ld_prior(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int2 ld_prior(const int2 *p) {   // 8 B aligned
    int2 v;
    asm volatile("ld.global.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ld_prior(const float2 *p) {   // 8 B aligned
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ int4 ld_prior(const int4 *p) {   // 16 B aligned
    int4 v;
    asm volatile("ld.global.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 ld_prior(const uint4 *p) {   // 16 B aligned
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ int32_t ld_l2(const int32_t *p) {
    int32_t v;
    asm volatile("ld.global.cg.s32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld_l2(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ int64_t ld_l2(const int64_t *p) {
    int64_t v;
    asm volatile("ld.global.cg.s64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ unsigned long long ld_l2(const unsigned long long *p) {
    unsigned long long v;
    asm volatile("ld.global.cg.u64 %0, [%1];" : "=l"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ ulonglong2 ld_l2(const ulonglong2 *p) {   // 16 B aligned
    ulonglong2 v;
    asm volatile("ld.global.cg.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p));
    return v;
}

}  // namespace dev
}  // namespace wk
