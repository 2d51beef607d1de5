// Values that one CTA hands over to another of the same launch, without flags or fences: a place of the workspace holds HANDED_EMPTY until its value is written, its one reader asks for
// it until it is there (bounded wait) and empties it again.  (A flag behind a fence costs the value two more trips to L2, and the writer the fence.)  A workspace is emptied when it is
// made and after a wait that ran out; launches that use it follow each other in one stream.
#pragma once
#include "common.cuh"

constexpr uint32_t HANDED_EMPTY = 0xffffffffu;      // as fp32 a NaN, which values never have: they would be handed over as another one

__device__ __forceinline__ uint32_t handed_bits(float v) { return __float_as_uint(v) == HANDED_EMPTY ? 0x7fffffffu : __float_as_uint(v); }
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t* p) {
    uint32_t v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ uint4 ld_relaxed(const uint4* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed(uint32_t* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ void st_relaxed(uint4* p, uint4 v) {
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}
