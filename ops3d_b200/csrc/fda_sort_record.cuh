// The list record of the cell-sorted backward, shared by the fill passes of attention and DCNv4.
#pragma once

#include <cuda_runtime.h>

namespace fda {

// One 32-byte list record as ONE streaming store (sm_100: 256-bit vector store); `rec` is 32-byte aligned.
__device__ __forceinline__ void store_record(float4 *rec, const float4 &a, const float4 &b) {
    asm volatile("st.global.cs.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(rec), "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w),
                 "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w) : "memory");
}

}  // namespace fda
